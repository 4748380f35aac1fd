// sweep_z.cu -- instantiations of the fused inviscid sweep along z
// (one translation unit per direction so the builds run in parallel).
#include <algorithm>

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
// An upper bound of sweep_z_blocks for every scheme and any owned planes of a
// grid: the marching kernel's segments hold a cell or more, the line kernel's
// C - 5 = 59, the chunked kernel's 8 - 5 = 3.
long sweep_z_blocks_max(long nx, long ny, long nz) {
    auto over = [](long a, long b) { return (a + b - 1) / b; };
    const long march = over(nx * ny, MARCH_NT) * nz;
    const long line = over(nx * ny, XL_WARPS) * over(nz, XLine<2, double>::C - 5);
    const long chunk = over(nx, SweepGeom<2, double>::NLINE) * ny * over(nz, SweepGeom<2, double>::C - 5);
    return std::max(march, std::max(line, chunk));
}
}  // namespace ns3d
