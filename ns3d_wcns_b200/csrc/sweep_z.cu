// sweep_z.cu -- instantiations of the fused inviscid sweep along z
// (one translation unit per direction so the builds run in parallel).
#include "sweep_line.cuh"

namespace ns3d {
cudaError_t sweep_z(const SweepArgs<double> &a, cudaStream_t st) {
    return !a.sp.char_recon ? line_or_march<2, double>(a, st) : sweep_char<2, double>(a, st);
}
cudaError_t sweep_z(const SweepArgs<float> &a, cudaStream_t st) {
    if (a.sp.char_recon) return sweep_char<2, float>(a, st);
    return a.L.nx & 1 || sweep32_scalar_forced() ? line_or_march<2, float>(a, st) : line_or_march<2, float2>(a, st);
}

// blocks of the z-sweep: the partials its fused stage 3 writes
long sweep_z_blocks(const SweepArgs<double> &a) {
    return !a.sp.char_recon ? line_or_march_blocks<2, double>(a) : sweep_blocks<2, double>(a);
}
long sweep_z_blocks(const SweepArgs<float> &a) {
    if (a.sp.char_recon) return sweep_blocks<2, float>(a);
    return a.L.nx & 1 || sweep32_scalar_forced() ? line_or_march_blocks<2, float>(a) : line_or_march_blocks<2, float2>(a);
}
}  // namespace ns3d
