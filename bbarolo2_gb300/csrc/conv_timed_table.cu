// The same with the tile table of MC models (conv_table.cu).
#include "conv_kernel.cuh"

void launch_conv_timed_table(cudaStream_t s, const GridDev &g, const MemberDev *mem, int nb, int maxt, int nzb, bool z16,
                             const float *model, long long mstride, int nz, const float *taps, int ky, int kx, int kxw,
                             float *smoothed, int do_conv, int do_resid, double *partial, int npart, TileSrc ts) {
    launch_widths<true, false>(s, g, mem, nb, maxt, nzb, z16, model, mstride, nz, taps, ky, kx, kxw, smoothed, do_conv,
                         do_resid, partial, npart, ts);
}
