// sweep_z.cu -- instantiations of the fused inviscid sweep along z
// (one translation unit per direction so the builds run in parallel).
#include "march.cuh"

namespace ns3d {
cudaError_t sweep_z(const SweepArgs<double> &a, cudaStream_t st) {
    return a.sp.char_recon ? sweep_select<2, double>(a, st) : march_select<2, double>(a, st);
}
cudaError_t sweep_z(const SweepArgs<float> &a, cudaStream_t st) { return sweep_select_f32<2>(a, st); }

// blocks of the z-sweep: the partials its fused stage 3 writes
long sweep_z_blocks(const SweepArgs<double> &a) {
    if (a.sp.char_recon) return (long)((a.L.nx + SweepGeom<2, double>::NLINE - 1) / SweepGeom<2, double>::NLINE) * a.L.ny;
    MarchArgs<double> m;
    const dim3 g = march_grid<2, double>(a, m);
    return (long)g.x * g.y;
}
}  // namespace ns3d
