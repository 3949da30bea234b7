// The ANALYTIC GALMOD deposit and the ring maps on the device (the reference's _galmod_analytic and
// _ring_maps_analytic, bbarolo/galmod.py:326-536).
//
//   k_an_model       any line, axis and layer: a warp a sample (sub-ring, radial sample, azimuth), lanes over heights, the
//                    runs of consecutive heights in one pixel found by ballots, their weights added in the
//                    reference's order, then the (run, channel) pairs over the lanes;
//   k_an_model_fast  sub-rings with one line on a linear axis (anfast), in float32: 32 samples set up a lane each;
//   k_an_records, k_an_amps, k_an_replay
//                    members that are member 0 but for the fluxes: its runs listed by pixel, read once for 16 members;
//   k_ant_bin, k_ant_list, k_ant_pixel
//                    thin disks (one height, anfast): the samples listed by pixel, a warp a pixel;
//   k_an_maps        ring maps: a run's weight in place of the line profile;
//   k_fix_to_model   fixed point to float32.
// What decides an index is the reference's: pixels and centre channels in float32 or float-float with a rounding bound,
// beyond it by the reference's float64 operations, each rounded once in its order (no contraction), so they are
// bit-exact. Values: k_an_model's and k_an_maps's are the reference's float64 ones; the float32 path's are within 1e-5 of
// the model's peak. The sums are in 64-bit fixed point (units 2^-e, e per member from a bound on its total flux):
// integer additions, exact and independent of the order of the deposits, so the model is deterministic; it differs from
// the reference's running float64 sum by rounding only.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "anpix.cuh"
#include "devmath.cuh"
#include "f32x2.cuh"
#include "kernels.h"

#define PHI_N 6146
#define AN_WPB 8            // warps per CTA
#define FULL 0xffffffffu

namespace {

// bbarolo/galmod.py:183-191: the normal CDF at t from the table (512 entries per unit from -6)
__device__ __forceinline__ double phi_interp(double t, const double *__restrict__ tab) {
    const double x = __dmul_rn(__dadd_rn(t, 6.0), 512.0);
    if (x <= 0.0) return 0.0;
    if (!(x < (double)(PHI_N - 1))) return 1.0;
    const int k = (int)x;
    const double t0 = tab[k], t1 = tab[k + 1];
    return __dadd_rn(t0, __dmul_rn(__dsub_rn(x, (double)k), __dsub_rn(t1, t0)));
}

// bbarolo/galmod.py:400-406: the pixel of the vertical sample at height z (z = 0 for a thin layer)
__device__ __forceinline__ void an_pixel(const AnSub &S, double cdelt0, double cdelt1, double xs, double xc,
                                         double yb, double z, int &g0, int &g1) {
    const double y = __dsub_rn(yb, __dmul_rn(z, S.sinc));
    g0 = clamp_pix(lround_ref(__dadd_rn(S.xpos, __ddiv_rn(__dsub_rn(xs, __dmul_rn(y, S.cpa)), cdelt0))));
    g1 = clamp_pix(lround_ref(__dadd_rn(S.ypos, __ddiv_rn(__dadd_rn(xc, __dmul_rn(y, S.spa)), cdelt1))));
}

// bbarolo/galmod.py:194-214: the CDF at the channel edges k0 .. k0 + nk of the line at velocity v (lanes over
// edges) into pe; the profile of channel k0 + j is |pe[j + 1] - pe[j]| * cd2i[k0 + j].
__device__ __forceinline__ void an_profile(const GridDev &g, int nl, double v, const AnSub &S,
                                           const double *__restrict__ vedges, const double *__restrict__ ptab,
                                           double *pe, int &k0, int &nk) {
    const int lane = threadIdx.x & 31;
    const long long kc = lround_ref(velgrid_exact(v, g, nl));
    long long a0 = kc - S.K, a1 = kc + S.K + 1;
    if (a0 < 0) a0 = 0;
    if (a1 > g.nz) a1 = g.nz;
    if (a1 <= a0) {
        k0 = 0;
        nk = 0;
        return;
    }
    k0 = (int)a0;
    nk = (int)(a1 - a0);
    const double *ve = vedges + (size_t)nl * (g.nz + 1) + k0;
    for (int j = lane; j <= nk; j += 32) pe[j] = phi_interp(__dmul_rn(__dsub_rn(ve[j], v), S.inv), ptab);
    __syncwarp();
}

// The channels of a profile times aw, added in fixed point to the spectrum o (whole warp).
__device__ __forceinline__ void an_add(unsigned long long *o, const double *pe, const double *__restrict__ cd2i,
                                       int k0, int nk, double aw, double fscale) {
    const int lane = threadIdx.x & 31;
    for (int j = lane; j < nk; j += 32) {
        double f = __dsub_rn(pe[j + 1], pe[j]);
        f = f >= 0 ? f : -f;
        const double t = __dmul_rn(aw, __dmul_rn(f, cd2i[k0 + j]));
        const long long q = __double2ll_rn(__dmul_rn(t, fscale));
        if (q) atomicAdd(o + k0 + j, (unsigned long long)q);
    }
}

// The runs of consecutive vertical samples in one pixel (bbarolo/galmod.py:412-421 and :518-524), in order:
// emit(g0, g1, ws) is called by the whole warp for each run (warp-uniform arguments).
template <class F>
__device__ __forceinline__ void an_runs(const AnSub &S, const double *__restrict__ zq, const double *__restrict__ wq,
                                        double cdelt0, double cdelt1, double xs, double xc, double yb, int *sgx,
                                        int *sgy, int *rg0, int *rg1, double *rws, F emit) {
    const int lane = threadIdx.x & 31;
    const int nzz = S.nzz;
    int og0 = 0, og1 = 0;
    double ows = 0.0;
    bool open = false;
    for (int base = 0; base < nzz; base += 32) {
        const int cnt = min(32, nzz - base);
        if (lane < cnt) {
            const double z = nzz > 1 ? __dmul_rn(zq[base + lane], S.z0) : 0.0;
            an_pixel(S, cdelt0, cdelt1, xs, xc, yb, z, sgx[lane], sgy[lane]);
        }
        __syncwarp();
        int nr = 0;
        if (lane == 0) {
            for (int t = 0; t < cnt; t++) {
                const int a = sgx[t], b = sgy[t];
                const double w = wq[base + t];
                if (open && a == og0 && b == og1) {
                    ows = __dadd_rn(ows, w);
                } else {
                    if (open) {
                        rg0[nr] = og0;
                        rg1[nr] = og1;
                        rws[nr] = ows;
                        nr++;
                    }
                    og0 = a;
                    og1 = b;
                    ows = w;
                    open = true;
                }
            }
        }
        nr = __shfl_sync(FULL, nr, 0);
        __syncwarp();
        for (int r = 0; r < nr; r++) emit(rg0[r], rg1[r], rws[r]);
        __syncwarp();
    }
    if (lane == 0) {
        rg0[0] = og0;
        rg1[0] = og1;
        rws[0] = ows;
    }
    __syncwarp();
    emit(rg0[0], rg1[0], rws[0]);
    __syncwarp();
}

struct AnWarp {
    int sgx[32], sgy[32], rg0[33], rg1[33];
    double rws[33];
};

// The (member, sample) of warp gs of a batch, by segments of warps: segment i (warps astart[i] .. astart[i + 1])
// is aseg[i] = (member whose model takes the deposits, member whose constants make them, sub-ring (-1: every
// sample of the table), sign of the deposits); s is the sample in the table.
struct AnSeg {
    int k, src, sign;
    long long s;
};
__device__ __forceinline__ bool an_seg(long long gs, const long long *__restrict__ astart,
                                       const int4 *__restrict__ aseg, int nseg, long long ntot,
                                       const int *__restrict__ sbase, AnSeg &o) {
    if (gs >= ntot) return false;
    int lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (astart[mid] <= gs) lo = mid;
        else hi = mid - 1;
    }
    const int4 sg = aseg[lo];
    o.k = sg.x;
    o.src = sg.y;
    o.sign = sg.w;
    o.s = gs - astart[lo] + (sg.z >= 0 ? sbase[sg.z] : 0);
    return true;
}

// The sample s of member src: sub-ring S, cos/sin of its azimuth; false if nothing to deposit.
__device__ __forceinline__ bool an_sample(long long s, int src, int nsub, const AnSub *__restrict__ subs,
                                          const int *__restrict__ sbase, const int *__restrict__ ssub,
                                          const double2 *__restrict__ cs, const AnSub *&S, double &caz,
                                          double &saz, double &R) {
    const int ir = ssub[s];
    S = subs + (size_t)src * nsub + ir;
    if (!S->active) return false;
    const int local = (int)(s - sbase[ir]);
    const double2 c = cs[s];
    caz = c.x;
    saz = c.y;
    R = S->R[local >= S->naz ? 1 : 0];
    return true;
}

// Models: out64 (per member: box (by, bx, nz), stride mstride) += fixed-point deposits. Every value is the reference's
// float64 one; what does not decide a value is kept off the float64 pipe (16 cycles of an SM an instruction): the
// pixels in float32 with a rounding bound (sample_pixel), the profile times cd2i once a sample and the amplitude times
// the run's weight, in fixed-point units (a power of two: exact), once a run, so that a deposit is one multiplication
// and one conversion, its (run, channel) pairs over the lanes. One 160x160x128 model: 3.6 ms with the pixels in
// float64, the runs found by one lane and four float64 operations a deposit, 1.42 ms so.
#define AN_RUNS 96
__global__ void __launch_bounds__(AN_WPB * 32) k_an_model(GridDev g, const AnSub *__restrict__ subs, int nsub,
                                                          const int *__restrict__ sbase, const int *__restrict__ ssub,
                                                          const double2 *__restrict__ cs,
                                                          const float2 *__restrict__ csf,
                                                          const long long *__restrict__ astart,
                                                          const int4 *__restrict__ aseg, int nseg, long long ntot,
                                                          const double *__restrict__ zq, const double *__restrict__ wq,
                                                          const float *__restrict__ zqf,
                                                          const double *__restrict__ vedges,
                                                          const double *__restrict__ cd2i,
                                                          const double *__restrict__ ptab,
                                                          const MemberDev *__restrict__ mem,
                                                          unsigned long long *__restrict__ out64, long long mstride,
                                                          int skip_fast) {
    extern __shared__ double an_smem[];
    __shared__ double rws[AN_WPB][AN_RUNS];                 // per warp: the runs of a sample (weight; pixel of the box)
    __shared__ int rpix[AN_WPB][AN_RUNS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long gs = (long long)blockIdx.x * AN_WPB + w;
    AnSeg sg;
    if (!an_seg(gs, astart, aseg, nseg, ntot, sbase, sg)) return;
    const int k = sg.k;
    const AnSub *Sp;
    double caz, saz, R;
    if (!an_sample(sg.s, sg.src, nsub, subs, sbase, ssub, cs, Sp, caz, saz, R)) return;
    const AnSub &S = *Sp;
    if (skip_fast && S.anfast) return;                 // (k_an_model_fast's samples)
    const double wside = caz >= 0.0 ? S.wrec : S.wapp;
    if (wside == 0.0) return;
    const MemberDev &M = mem[k];
    const int nz = g.nz, nl_n = g.nlines;
    double *pe = an_smem + (size_t)w * nl_n * (nz + 2);
    // (a negative unit: the deposits of member 0's constants taken out of a difference, rounded symmetrically)
    const double fscale = sg.sign < 0 ? -ldexp(1.0, M.fix_exp) : ldexp(1.0, M.fix_exp);
    unsigned long long *o64 = out64 + (size_t)k * mstride;
    // bbarolo/galmod.py:407
    const double vplane = __dadd_rn(__dadd_rn(S.vsys, __dmul_rn(__dadd_rn(__dmul_rn(S.vrot, caz), __dmul_rn(S.vrad, saz)),
                                                                S.sinc)),
                                    __dmul_rn(S.vvert, S.cinc));
    const double *zqs = zq + S.zq_off, *wqs = wq + S.zq_off;
    if (!S.zdep) {
        const int nzz = S.nzz, kr = (int)(sg.s - sbase[ssub[sg.s]]) >= S.naz ? 1 : 0;
        const PixF px = pix_setup(S, kr, csf[sg.s], zqf + S.zq_off, nzz);
        const double2 *cp = cs + sg.s;
        bool ready = false;
        int lk0[BBGPU_MAXL], lnk[BBGPU_MAXL];
        auto deposit = [&](int n) {                    // the n runs of the list (bbarolo/galmod.py:422-428)
            if (!ready) {
                for (int nl = 0; nl < nl_n; nl++) {
                    double *f = pe + (size_t)nl * (nz + 2);
                    an_profile(g, nl, vplane, S, vedges, ptab, f, lk0[nl], lnk[nl]);
                    // (the profile in place of the CDF: a lane's value before the next lane's edge is overwritten)
                    for (int j0 = 0; j0 < lnk[nl]; j0 += 32) {
                        const int j = j0 + lane;
                        double v = 0.0;
                        if (j < lnk[nl]) v = __dmul_rn(fabs(__dsub_rn(f[j + 1], f[j])), cd2i[lk0[nl] + j]);
                        __syncwarp();
                        if (j < lnk[nl]) f[j] = v;
                        __syncwarp();
                    }
                }
                ready = true;
            }
            for (int nl = 0; nl < nl_n; nl++) {
                const int nk = lnk[nl];
                if (nk == 0) continue;
                const double *f = pe + (size_t)nl * (nz + 2);
                const double aw0 = __dmul_rn(S.a[nl], wside);
                double aw[AN_RUNS / 32];
#pragma unroll
                for (int i = 0; i < AN_RUNS / 32; i++)
                    aw[i] = i * 32 + lane < n ? __dmul_rn(__dmul_rn(aw0, rws[w][i * 32 + lane]), fscale) : 0.0;
                int r = 0, j = lane;
                while (j >= nk) {
                    j -= nk;
                    r++;
                }
                for (int i0 = 0; i0 < n * nk; i0 += 32) {
                    double a = __shfl_sync(FULL, aw[0], r & 31);
#pragma unroll
                    for (int i = 1; i < AN_RUNS / 32; i++) {
                        const double b = __shfl_sync(FULL, aw[i], r & 31);
                        if ((r >> 5) == i) a = b;
                    }
                    if (r < n) {
                        const long long q = __double2ll_rn(__dmul_rn(a, f[j]));
                        if (q) atomicAdd(o64 + (size_t)rpix[w][r] * nz + lk0[nl] + j, (unsigned long long)q);
                    }
                    j += 32;
                    while (j >= nk) {
                        j -= nk;
                        r++;
                    }
                }
            }
        };
        bool open = false;                             // a run carried from the previous pass
        int cg0 = 0, cg1 = 0, nr = 0;
        double cws = 0.0;
        for (int base = 0; base < nzz; base += 32) {
            const int cnt = min(32, nzz - base);
            const bool valid = lane < cnt;
            int g0 = 0x7fffffff, g1 = 0x7fffffff;
            if (valid)
                sample_pixel(S, px, kr, cp, nzz, nzz > 1 ? zqf[S.zq_off + base + lane] : 0.f, zqs + base + lane, g.cdelt0,
                             g.cdelt1, g0, g1);
            const int pg0 = __shfl_up_sync(FULL, g0, 1), pg1 = __shfl_up_sync(FULL, g1, 1);
            const bool start = valid && (lane == 0 ? (!open || g0 != cg0 || g1 != cg1) : (g0 != pg0 || g1 != pg1));
            const unsigned smask = __ballot_sync(FULL, start);
            if (open && (smask & 1u)) {                // the carried run ended with the previous pass
                const int rx = cg0 - M.blo0, ry = cg1 - M.blo1;
                if ((unsigned)rx < (unsigned)M.bx && (unsigned)ry < (unsigned)M.by) {
                    if (lane == 0) {
                        rpix[w][nr] = ry * M.bx + rx;
                        rws[w][nr] = cws;
                    }
                    nr++;
                }
                open = false;
            }
            const bool last = lane == cnt - 1, final_pass = base + 32 >= nzz;
            const bool end = valid && (last || ((smask >> (lane + 1)) & 1u));
            // the run's weight, its heights added in their order (bbarolo/galmod.py:416-418)
            const unsigned upto = smask & (0xffffffffu >> (31 - lane));
            double ws = 0.0;
            if (end) {
                int t = 0;
                if (upto) {
                    t = 31 - __clz(upto);
                    ws = wqs[base + t++];
                } else {
                    ws = cws;
                }
                for (; t <= lane; t++) ws = __dadd_rn(ws, wqs[base + t]);
            }
            const int rx = g0 - M.blo0, ry = g1 - M.blo1;
            const bool put = end && (!last || final_pass) && (unsigned)rx < (unsigned)M.bx && (unsigned)ry < (unsigned)M.by;
            const unsigned pmask = __ballot_sync(FULL, put);
            if (put) {
                const int at = nr + __popc(pmask & ((1u << lane) - 1u));
                rpix[w][at] = ry * M.bx + rx;
                rws[w][at] = ws;
            }
            nr += __popc(pmask);
            if (nr > 0 && (final_pass || nr > AN_RUNS - 33)) {
                __syncwarp();
                deposit(nr);
                __syncwarp();
                nr = 0;
            }
            if (!final_pass) {
                cg0 = __shfl_sync(FULL, g0, cnt - 1);
                cg1 = __shfl_sync(FULL, g1, cnt - 1);
                cws = __shfl_sync(FULL, ws, cnt - 1);
                open = true;
            }
        }
        return;
    }
    const double x = __dmul_rn(R, caz);
    const double yb = __dmul_rn(__dmul_rn(R, saz), S.cinc);
    const double xs = __dmul_rn(x, S.spa), xc = __dmul_rn(x, S.cpa);
    // bbarolo/galmod.py:430-463: the velocity depends on |z|; the samples at +z and -z share a profile
    const int nzz = S.nzz;
    for (int kz = 0; kz < (nzz + 1) / 2; kz++) {
        const int kz2 = nzz - 1 - kz;
        int ga = 0, gb = 0;
        if (lane < 2) {
            const double z = __dmul_rn(zqs[lane == 0 ? kz : kz2], S.z0);
            an_pixel(S, g.cdelt0, g.cdelt1, xs, xc, yb, z, ga, gb);
        }
        const int gx1 = __shfl_sync(FULL, ga, 0), gy1 = __shfl_sync(FULL, gb, 0);
        const int gx2 = __shfl_sync(FULL, ga, 1), gy2 = __shfl_sync(FULL, gb, 1);
        const bool in1 = !(gx1 < M.blo0 || gx1 >= M.bhi0 || gy1 < M.blo1 || gy1 >= M.bhi1);
        const bool in2 = kz2 != kz && !(gx2 < M.blo0 || gx2 >= M.bhi0 || gy2 < M.blo1 || gy2 >= M.bhi1);
        if (!(in1 || in2)) continue;
        const double az_ = fabs(__dmul_rn(zqs[kz], S.z0));
        double v = vplane;
        if (az_ > S.zcyl) {
            const double lv = __dsub_rn(S.vrot, __dmul_rn(S.dvdz, __dsub_rn(az_, S.zcyl)));
            const double vr = S.vrot >= 0.0 ? ((0.0 > lv) ? 0.0 : lv) : ((0.0 < lv) ? 0.0 : lv);
            v = __dadd_rn(__dadd_rn(S.vsys, __dmul_rn(__dadd_rn(__dmul_rn(vr, caz), __dmul_rn(S.vrad, saz)), S.sinc)),
                          __dmul_rn(S.vvert, S.cinc));
        }
        for (int nl = 0; nl < nl_n; nl++) {
            int k0, nk;
            an_profile(g, nl, v, S, vedges, ptab, pe, k0, nk);
            if (nk == 0) continue;
            const double a = __dmul_rn(S.a[nl], wside);
            if (in1 && in2 && gx1 == gx2 && gy1 == gy2) {
                unsigned long long *o = o64 + ((size_t)(gy1 - M.blo1) * M.bx + (size_t)(gx1 - M.blo0)) * nz;
                an_add(o, pe, cd2i, k0, nk, __dmul_rn(a, __dadd_rn(wqs[kz], wqs[kz2])), fscale);
            } else {
                if (in1) {
                    unsigned long long *o = o64 + ((size_t)(gy1 - M.blo1) * M.bx + (size_t)(gx1 - M.blo0)) * nz;
                    an_add(o, pe, cd2i, k0, nk, __dmul_rn(a, wqs[kz]), fscale);
                }
                if (in2) {
                    unsigned long long *o = o64 + ((size_t)(gy2 - M.blo1) * M.bx + (size_t)(gx2 - M.blo0)) * nz;
                    an_add(o, pe, cd2i, k0, nk, __dmul_rn(a, wqs[kz2]), fscale);
                }
            }
            __syncwarp();
        }
    }
}

// ------------------------------------------------------------------------------ the model's float32 path
// Sub-rings with one line on a linear channel map and a velocity independent of the height (anfast), for each
// (member, azimuth sample):
//   pixels  lanes over heights, float32 with a rounding bound and exact fallbacks (sample_pixel), the reference's
//           pixel of every height;
//   runs    consecutive heights in one pixel (a ballot of the run starts), their weights by a segmented scan
//           (float32), a run crossing a pass of 32 heights carried to the next pass;
//   line    the velocity and its channel in float-float (the reference's
//           float64 _velgrid within 1e-6 of a channel boundary), the centre channel kc exact, then the
//           channel-integrated profile over kc - K .. kc + K in float32: the edges relative to a reference
//           velocity in float-float (so that (edge - v) / sig keeps ~1e-7), the normal CDF from the reference's
//           table (float32 copy, linear interpolation as _phi);
//   deposit lanes over channels, 64-bit fixed-point atomics of profile x amplitude x run weight (float32
//           products, each rounded to the unit 2^-e: exact and order-independent sums).
#define ANF_WPB 8

// (the integer part by an addition rounded down: the conversion instructions run at an eighth of the float32 rate;
// no branch: outside the table the index is clamped and the value replaced)
__device__ __forceinline__ float phi_f32(float t, const float *__restrict__ tab) {
    const float x = (t + 6.0f) * 512.0f;
    const float y = fminf(fmaxf(x, 0.0f), 6144.9995f);              // (the largest float32 below the last entry)
    const float f = __fadd_rd(y, 8388608.0f);
    const int k = __float_as_int(f) - 0x4B000000;
    const float t0 = tab[k], t1 = tab[k + 1];
    const float v = fmaf(y - __fsub_rn(f, 8388608.0f), t1 - t0, t0);
    return !(x > 0.0f) ? 0.0f : (x >= (float)(PHI_N - 1) ? 1.0f : v);
}

// The line of a float32-path sample: bbarolo/galmod.py:407 and :410 (_velgrid, _lround) in float-float (about 44
// bits: the channel and the velocity relative to vref within ~1e-11 of the reference's float64 values); within 1e-6
// of a channel boundary the reference's float64 operations decide the centre channel. Returns the centre channel
// and the line-of-sight velocity v (float-float).
__device__ __forceinline__ long long fast_line_centre(const AnSub &S, const GridDev &g, float4 cq,
                                                      const double2 *__restrict__ cp, ff &v) {
    const ff caz{cq.x, cq.y}, saz{cq.z, cq.w};
    v = ff_add(ff_mul(ff{S.vroth, S.vrotl}, caz), ff_mul(ff{S.vradh, S.vradl}, saz));
    v = ff_add(ff_mul(v, ff{S.sinch, S.sincl}), ff_mul(ff{S.vverth, S.vvertl}, ff{S.cinch, S.cincl}));
    v = ff_add(ff{S.vsysh, S.vsysl}, v);
    const ff chd = ff_add(ff_mul(v, ff{g.ia0h, g.ia0l}), ff{g.ib0h, g.ib0l});
    int kci;
    if (ff_round(chd, kci)) return kci;
    const double2 c = *cp;
    const double vplane = __dadd_rn(__dadd_rn(S.vsys, __dmul_rn(__dadd_rn(__dmul_rn(S.vrot, c.x),
                                                                          __dmul_rn(S.vrad, c.y)), S.sinc)),
                                    __dmul_rn(S.vvert, S.cinc));
    return lround_ref(velgrid_exact(vplane, g, 0));
}

// The float32 nearest to q 2^-e: the two 23-bit halves of |q| < 2^46 are exact in float32 and joined by one FMA, so
// there is one rounding and no float64 conversion (the float64 route, 3 instructions of the 1/64-rate pipe, held the
// conversion of the models to 190 G values/s). Larger sums are shifted down first, the bits lost kept as a sticky one.
__device__ __forceinline__ float fix_to_f32(long long q, int e) {
    unsigned long long m = q < 0 ? 0ULL - (unsigned long long)q : (unsigned long long)q;
    int x = -e;
    if (m >> 46) {
        m = (m >> 18) | ((m & 0x3ffffULL) != 0);
        x += 18;
    }
    const float hi = __fsub_rn(__int_as_float(0x4B000000 | (int)(m >> 23)), 8388608.0f);
    const float lo = __fsub_rn(__int_as_float(0x4B000000 | ((int)m & 0x7fffff)), 8388608.0f);
    const float f = fmaf(hi, 8388608.0f, lo);
    // (a power of two or a product outside the normal range: ldexpf's own rounding)
    const float r = x > -126 && x < 80 ? __fmul_rn(f, __int_as_float((x + 127) << 23)) : ldexpf(f, x);
    return q < 0 ? -r : r;
}

// What a warp needs of one of its 32 samples, staged in shared memory by the lane that set the sample up.
struct __align__(16) AnfSample {
    float vrh, vrl, invf, amp;        // the line: velocity about vref (float-float), 1 / sig, fixed-point amplitude
    float bxf, byf, zP3, zQ3;         // the pixels (PixF); hwx < 0: every height takes the exact path
    float hwx, hwy;
    unsigned short k0, nk;            // the line's channels (an_smem_bytes keeps nz far below 65536)
    int off;                          // the vertical samples
    int nzz, sub, s, k;               // their number; index of the constants; sample (bit 31: second radius); member
};

#define ANF_RUNS 96                   // runs of a sample collected before their deposit (a pass adds at most 33)
#define ANF_FIXMAX 1.7592186044416e13f // 2^44: below it f32_to_fix is f32_to_ll

// f32_to_ll for |x| < ANF_FIXMAX without its branch and shift: adding 1.5 2^46 rounded down leaves the multiple of 2^23
// below x in the low mantissa bits of t, and the rest, at most 2^23, is rounded to an integer in the low bits of q.
#define ANF_HI 1.0555311626649600e14f    // 1.5 2^46
#define ANF_TOP (ANF_HI + 8388608.0f)    // (exact: 24 bits)
__device__ __forceinline__ unsigned long long f32_to_fix(float x) {
    const float t = __fadd_rd(x, ANF_HI);
    const float q = __fadd_rn(x, __fsub_rn(ANF_TOP, t));
    return (unsigned long long)((long long)(__float_as_int(t) - __float_as_int(ANF_HI)) * 8388608 +
                                (__float_as_int(q) - 0x4B000000));
}

// The set-up of sample s (constants S = subs[sub], radius kr) by its lane; false if its line has no channel in the band.
__device__ __forceinline__ bool anf_setup(const GridDev &g, const AnSub &S, int sub, int s, int kr, float2 cf,
                                          const float4 *__restrict__ csff, const double2 *__restrict__ cs,
                                          const float *__restrict__ zqf, AnfSample &o) {
    ff v;
    const long long kc = fast_line_centre(S, g, csff[s], cs + s, v);
    long long a0 = kc - S.K, a1 = kc + S.K + 1;
    if (a0 < 0) a0 = 0;
    if (a1 > g.nz) a1 = g.nz;
    if (a1 <= a0) return false;
    const PixF px = pix_setup(S, kr, cf, zqf + S.zq_off, S.nzz);
    const ff vr = ff_add(v, ff{-g.vrefh, -g.vrefl});
    o.vrh = vr.hi;
    o.vrl = vr.lo;
    o.invf = S.invf;
    o.bxf = px.bxf;
    o.byf = px.byf;
    o.zP3 = px.zP3;
    o.zQ3 = px.zQ3;
    o.hwx = px.fast ? px.hwx : -1.0f;
    o.hwy = px.hwy;
    o.k0 = (unsigned short)a0;
    o.nk = (unsigned short)(a1 - a0);
    o.off = S.zq_off;
    o.nzz = S.nzz;
    o.sub = sub;
    o.s = s | (kr << 31);
    return true;
}

// The runs of a sample's heights in the box (bw, bh from blo0, blo1), 32 heights a pass, collected in the warp's list
// run (pixel, weight); flush(n) takes the n of a full list and the last ones.
template <class F>
__device__ __forceinline__ void anf_runs(const GridDev &g, const AnfSample &o, const AnSub &S,
                                         const double2 *__restrict__ cs, const double *__restrict__ zq,
                                         const float *__restrict__ zqf, const float *__restrict__ wqf, int blo0,
                                         int blo1, int bw, int bh, int lane, int2 *run, F flush) {
    const PixF px{o.bxf, o.byf, o.zP3, o.zQ3, o.hwx, o.hwy, o.hwx > 0.0f};
    const int nzz = o.nzz, off = o.off;
    const double2 *cp = cs + (o.s & 0x7fffffff);
    const int kr = (unsigned)o.s >> 31;
    bool open = false;                                  // a run carried from the previous pass
    int cg0 = 0, cg1 = 0, nr = 0;
    float cws = 0.0f;
    for (int base = 0; base < nzz; base += 32) {
        const int cnt = min(32, nzz - base);
        const bool valid = lane < cnt;
        int g0 = 0x7fffffff, g1 = 0x7fffffff;
        float wv = 0.0f;
        if (valid) {
            sample_pixel(S, px, kr, cp, nzz, nzz > 1 ? __ldg(zqf + off + base + lane) : 0.f,
                         zq + off + base + lane, g.cdelt0, g.cdelt1, g0, g1);
            wv = __ldg(wqf + off + base + lane);
        }
        const int pg0 = __shfl_up_sync(FULL, g0, 1), pg1 = __shfl_up_sync(FULL, g1, 1);
        const bool start = valid && (lane == 0 ? (!open || g0 != cg0 || g1 != cg1) : (g0 != pg0 || g1 != pg1));
        const unsigned smask = __ballot_sync(FULL, start);
        if (open && (smask & 1u)) {                     // the carried run ended with the previous pass
            const int rx = cg0 - blo0, ry = cg1 - blo1;
            if ((unsigned)rx < (unsigned)bw && (unsigned)ry < (unsigned)bh) {
                if (lane == 0) run[nr] = make_int2(ry * bw + rx, __float_as_int(cws));
                nr++;
            }
            open = false;
        }
        // segmented inclusive scan of the weights (a segment: from a run start to the lane before the next)
        const unsigned upto = smask & (0xffffffffu >> (31 - lane));
        const int head = upto ? 31 - __clz(upto) : 0;
        float v = wv;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float t = __shfl_up_sync(FULL, v, d);
            if (lane - d >= head) v += t;
        }
        if (!upto && open) v += cws;                    // (the lanes that continue the carried run)
        const bool nstart = lane < 31 && ((smask >> (lane + 1)) & 1u);
        const bool last = lane == cnt - 1;
        const bool final_pass = base + 32 >= nzz;
        const bool done = valid && ((!last && nstart) || (last && final_pass));
        const int rx = g0 - blo0, ry = g1 - blo1;
        const bool put = done && (unsigned)rx < (unsigned)bw && (unsigned)ry < (unsigned)bh;
        const unsigned pmask = __ballot_sync(FULL, put);
        if (put) run[nr + __popc(pmask & ((1u << lane) - 1u))] = make_int2(ry * bw + rx, __float_as_int(v));
        nr += __popc(pmask);
        if (final_pass || nr > ANF_RUNS - 33) {
            __syncwarp();
            flush(nr);
            __syncwarp();
            nr = 0;
        }
        if (!final_pass) {
            cg0 = __shfl_sync(FULL, g0, cnt - 1);
            cg1 = __shfl_sync(FULL, g1, cnt - 1);
            cws = __shfl_sync(FULL, v, cnt - 1);
            open = true;
        }
    }
}

// The samples are set up 32 at a time, a lane each (constants, pixel coefficients, line); then the warp takes them one
// after another: the profile over the lanes into shared memory; the heights, 32 a pass, into the list of the sample's
// runs in the box; and the (run, channel) pairs laid end to end over the lanes, one 64-bit reduction each. At 27
// channels and 20 runs that is about 550 instructions a sample, where a warp that set up and deposited a run at a time
// took 1200 (40 ms for the thick gradient of 161 members, 160x160x128).
__global__ void __launch_bounds__(ANF_WPB * 32, 4) k_an_model_fast(GridDev g, const AnSub *__restrict__ subs, int nsub,
                                                                const int *__restrict__ sbase,
                                                                const int *__restrict__ ssub,
                                                                const double2 *__restrict__ cs,
                                                                const float2 *__restrict__ csf,
                                                                const float4 *__restrict__ csff,
                                                                const long long *__restrict__ astart,
                                                                const int4 *__restrict__ aseg, int nseg,
                                                                long long ntot, const double *__restrict__ zq,
                                                                const float *__restrict__ zqf,
                                                                const float *__restrict__ wqf,
                                                                const float2 *__restrict__ vef,
                                                                const float *__restrict__ cd2if,
                                                                const float *__restrict__ ptabf,
                                                                const MemberDev *__restrict__ mem,
                                                                unsigned long long *__restrict__ out64,
                                                                long long mstride) {
    extern __shared__ __align__(16) uint8_t anf_smem[];     // samples, runs, the CDF table, profiles
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nz = g.nz;
    AnfSample *const sm = (AnfSample *)anf_smem + w * 32;
    int2 *const run = (int2 *)(anf_smem + ANF_WPB * 32 * sizeof(AnfSample)) + w * ANF_RUNS;
    float *const tab = (float *)(anf_smem + ANF_WPB * (32 * sizeof(AnfSample) + ANF_RUNS * sizeof(int2)));
    float *const prof = tab + PHI_N + w * nz;
    // (the lanes' channel edges are ~100 entries of the table apart: a gather, cheap in shared memory)
    for (int i = threadIdx.x; i < PHI_N; i += ANF_WPB * 32) tab[i] = ptabf[i];
    __syncthreads();
    const long long gs = ((long long)blockIdx.x * ANF_WPB + w) * 32 + lane;
    bool ok = false;
    AnSeg sg;
    if (an_seg(gs, astart, aseg, nseg, ntot, sbase, sg)) {
        const int s = (int)sg.s, ir = ssub[s];
        const AnSub &S = subs[(size_t)sg.src * nsub + ir];
        const float2 cf = csf[s];
        const bool rec = cf.x >= 0.0f;                      // (the sign of the float32 table is the float64 test's)
        if (S.active && S.anfast && !(S.wzero & (rec ? 1 : 2))) {
            ok = anf_setup(g, S, sg.src * nsub + ir, s, s - sbase[ir] >= S.naz ? 1 : 0, cf, csff, cs, zqf, sm[lane]);
            if (ok) {
                sm[lane].amp = (float)sg.sign * ldexpf(S.af * (rec ? S.wrecf : S.wappf), mem[sg.k].fix_exp);
                sm[lane].k = sg.k;
            }
        }
    }
    unsigned todo = __ballot_sync(FULL, ok);
    __syncwarp();
    for (; todo; todo &= todo - 1) {
        const AnfSample &o = sm[__ffs(todo) - 1];
        const int nk = o.nk, k0 = o.k0;
        const AnSub &S = subs[o.sub];
        const MemberDev &M = mem[o.k];
        const int blo0 = M.blo0, blo1 = M.blo1, bw = M.bx, bh = M.by;
        unsigned long long *const o64 = out64 + (size_t)o.k * mstride + k0;
        // the profile: a lane's upper edge is the next lane's lower one
        bool big = false;
        for (int j = lane; j - lane < nk; j += 31) {
            const float2 e = __ldg(vef + k0 + min(j, nk));
            const float ph = phi_f32((__fsub_rn(e.x, o.vrh) + __fsub_rn(e.y, o.vrl)) * o.invf, tab);
            const float pn = __shfl_down_sync(FULL, ph, 1);
            if (lane < 31 && j < nk) {
                const float p = fabsf(pn - ph) * __ldg(cd2if + k0 + j) * o.amp;
                prof[j] = p;
                big |= !(fabsf(p) < 0.5f * ANF_FIXMAX);                          // (a weight is at most about 1)
            }
        }
        big = __any_sync(FULL, big);
        // the n runs of the list, their (run, channel) pairs over the lanes: 32 pairs on are dr runs and dj channels
        int r0 = 0, j0 = lane, dr = 0, dj = 32;
        while (j0 >= nk) {
            j0 -= nk;
            r0++;
        }
        while (dj >= nk) {
            dj -= nk;
            dr++;
        }
        auto deposit = [&](int n) {
            const int2 *e = run + r0;
            const int2 *const end = run + n;
            int j = j0;
            if (!big) {
                while (e < end) {
                    const int2 q = *e;
                    atomicAdd(o64 + j + (long long)q.x * nz, f32_to_fix(prof[j] * __int_as_float(q.y)));
                    j += dj;
                    e += dr;
                    if (j >= nk) {
                        j -= nk;
                        e++;
                    }
                }
            } else {
                while (e < end) {
                    const int2 q = *e;
                    atomicAdd(o64 + j + (long long)q.x * nz,
                              (unsigned long long)f32_to_ll(prof[j] * __int_as_float(q.y)));
                    j += dj;
                    e += dr;
                    if (j >= nk) {
                        j -= nk;
                        e++;
                    }
                }
            }
        };
        anf_runs(g, o, S, cs, zq, zqf, wqf, blo0, blo1, bw, bh, lane, run, deposit);
    }
}

// ------------------------------------------------------------------ members that are member 0 but for the fluxes
// A member whose sub-rings are member 0's but for the density (a step of a geometry parameter of one ring, whose flux
// normalisation moves every ring's) has member 0's runs and profiles: only the amplitudes differ. Member 0's runs are
// listed by pixel and block of 32 channels beside the profiles of their samples (k_an_records: counted, then placed),
// and a warp takes a list and 16 members: it reads each run and its profile once and adds the 16 members' deposits in
// registers. The deposits are k_an_model_fast's, integer for integer, without its reductions in L2 (15 SM cycles a
// warp of deposits against 3); the model is written in float32. The sub-rings that differ are deposited by
// k_an_model_fast beforehand and added here. Bound by the float32 pipe (five packed operations for two deposits) and
// the issue slots: 80 members of 160x160x128 4.8 ms, against 12.2 ms by their samples; with 64-bit sums 6.9 ms, with
// six operations and single runs 6.6 ms.
struct __align__(16) AnRun {
    int s;                // the sample, whose profile is prof[s kw ..]
    float w;              // the weight of the run
    unsigned kn;          // first channel | channels << 16
    unsigned hb;          // 2 sub-ring + (receding 0, approaching 1) | upper half: a bound of profile x weight (a
                          // bfloat16, rounded up)
};
#define ANR_MG 16                     // members of a warp
#define ANR_D 8                       // profiles on their way

template <bool PLACE>
__global__ void __launch_bounds__(ANF_WPB * 32) k_an_records(GridDev g, const AnSub *__restrict__ subs,
                                                             const int *__restrict__ sbase,
                                                             const int *__restrict__ ssub,
                                                             const double2 *__restrict__ cs,
                                                             const float2 *__restrict__ csf,
                                                             const float4 *__restrict__ csff, long long ns,
                                                             const unsigned long long *__restrict__ act,
                                                             const double *__restrict__ zq,
                                                             const float *__restrict__ zqf,
                                                             const float *__restrict__ wqf,
                                                             const float2 *__restrict__ vef,
                                                             const float *__restrict__ cd2if,
                                                             const float *__restrict__ ptabf,
                                                             const MemberDev *__restrict__ mem, int *__restrict__ count,
                                                             AnRun *__restrict__ runs, float *__restrict__ prof,
                                                             int kw) {
    __shared__ AnfSample sm_[ANF_WPB][32];
    __shared__ int2 run_[ANF_WPB][ANF_RUNS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    AnfSample *const sm = sm_[w];
    int2 *const run = run_[w];
    const long long s0 = ((long long)blockIdx.x * ANF_WPB + w) * 32 + lane;
    bool ok = false;
    if (s0 < ns) {
        const int s = (int)s0, ir = ssub[s];
        const AnSub &S = subs[ir];
        const float2 cf = csf[s];
        const int half = cf.x >= 0.0f ? 0 : 1;
        if (((act[ir >> 6] >> (ir & 63)) & 1ull) && !(S.wzero & (1 << half))) {
            ok = anf_setup(g, S, ir, s, s - sbase[ir] >= S.naz ? 1 : 0, cf, csff, cs, zqf, sm[lane]);
            sm[lane].k = 2 * ir + half;
        }
    }
    const MemberDev &M = mem[0];
    const int blo0 = M.blo0, blo1 = M.blo1, bw = M.bx, bh = M.by, nzb = (g.nz + 31) / 32;
    unsigned todo = __ballot_sync(FULL, ok);
    __syncwarp();
    for (; todo; todo &= todo - 1) {
        const AnfSample &o = sm[__ffs(todo) - 1];
        const int nk = o.nk, k0 = o.k0, s = o.s & 0x7fffffff;
        float top = 0.0f;
        if (PLACE) {
            for (int j = lane; j - lane < nk; j += 31) {    // (the profile as k_an_model_fast's, before the amplitude)
                const float2 e = __ldg(vef + k0 + min(j, nk));
                const float ph = phi_f32((__fsub_rn(e.x, o.vrh) + __fsub_rn(e.y, o.vrl)) * o.invf, ptabf);
                const float pn = __shfl_down_sync(FULL, ph, 1);
                if (lane < 31 && j < nk) {
                    const float p = fabsf(pn - ph) * __ldg(cd2if + k0 + j);
                    prof[(size_t)s * kw + j] = p;
                    top = fmaxf(top, fabsf(p));
                }
            }
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) top = fmaxf(top, __shfl_xor_sync(FULL, top, d));
        }
        anf_runs(g, o, subs[o.sub], cs, zq, zqf, wqf, blo0, blo1, bw, bh, lane, run, [&](int n) {
            for (int r = lane; r < n; r += 32) {
                const int2 q = run[r];
                const float w = __int_as_float(q.y);
                const unsigned b = (__float_as_uint(top * fabsf(w)) & 0xffff0000u) + 0x10000u;
                for (int zb = k0 >> 5; zb <= (k0 + nk - 1) >> 5; zb++) {
                    const int at = atomicAdd(count + q.x * nzb + zb, 1);
                    if (PLACE) runs[at] = AnRun{s, w, (unsigned)k0 | ((unsigned)nk << 16), (unsigned)o.k | b};
                }
            }
        });
    }
}

// The members' amplitudes of (sub-ring, side): amp[2 sub-ring + side][member of klist] (padded to ANR_MG; 0 where the
// member deposits the sub-ring itself, chg, or has none), and the largest of each group of ANR_MG.
__global__ void k_an_amps(const AnSub *__restrict__ subs, int nsub, const MemberDev *__restrict__ mem,
                          const int *__restrict__ klist, int n3, int ng, const unsigned long long *__restrict__ chg,
                          int nchw, float *__restrict__ amp, float *__restrict__ top) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int np = ng * ANR_MG, ih = (int)(i / np), m = (int)(i - (long long)ih * np), ir = ih >> 1;
    float a = 0.0f;
    if (ir < nsub && m < n3) {
        const int k = klist[m];
        const AnSub &S = subs[(size_t)k * nsub + ir];
        if (S.active && !((chg[(size_t)m * nchw + (ir >> 6)] >> (ir & 63)) & 1ull) && !(S.wzero & (1 << (ih & 1))))
            a = ldexpf(S.af * ((ih & 1) ? S.wappf : S.wrecf), mem[k].fix_exp);
    }
    float t = fabsf(a);
#pragma unroll
    for (int d = ANR_MG / 2; d > 0; d >>= 1) t = fmaxf(t, __shfl_xor_sync(FULL, t, d));
    if (ir >= nsub) return;
    amp[i] = a;
    if (m % ANR_MG == 0) top[(size_t)ih * ng + m / ANR_MG] = t;
}

// f32_to_fix of two values x (|x| < ANF_FIXMAX / 2, packed float32 operations): t holds the multiple of 2^23 below x in
// its low mantissa bits, q the rest rounded to an integer of at most 2^23. Sums of both stay within 32 bits for ANR_FLUSH
// runs, each addition with the bias of its constant.
#define ANR_FLUSH 256
__device__ __forceinline__ void fix_parts(unsigned long long x, unsigned long long &t, unsigned long long &q) {
    t = f32x2_add_rm(x, f32x2(ANF_HI, ANF_HI));
    q = f32x2_add(x, f32x2_fma(t, f32x2(-1.0f, -1.0f), f32x2(ANF_TOP, ANF_TOP)));
}

// A CTA keeps the amplitudes of one group of members in shared memory and its warps take (pixel, 32 channels) after
// (pixel, 32 channels).
__global__ void __launch_bounds__(256, 3) k_an_replay(int nz, int ng, int nzb, int npix, int ntask, int na,
                                                      const int *__restrict__ offset, const int *__restrict__ count,
                                                      const int4 *__restrict__ runs, const float *__restrict__ prof,
                                                      int kw, const float *__restrict__ amp,
                                                      const float *__restrict__ top, const int *__restrict__ klist,
                                                      int n3, const MemberDev *__restrict__ mem,
                                                      const unsigned long long *__restrict__ own, long long mstride,
                                                      float *__restrict__ model) {
    extern __shared__ __align__(16) float anr_amp[];        // na x ANR_MG amplitudes, na bounds
    __shared__ unsigned long long sum_[8][ANR_MG][32];      // sums beyond 32 bits, where there are any
    __shared__ float ring_[8][ANR_D][32];                   // the profiles of the next runs
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = blockIdx.x % ng;
    float *const atop = anr_amp + na * ANR_MG;
    for (int i = threadIdx.x; i < na * ANR_MG; i += 256)
        anr_amp[i] = __ldg(amp + ((size_t)(i / ANR_MG) * ng + grp) * ANR_MG + i % ANR_MG);
    for (int i = threadIdx.x; i < na; i += 256) atop[i] = __ldg(top + (size_t)i * ng + grp);
    __syncthreads();
    unsigned long long (*const sum)[32] = sum_[warp];
    float (*const ring)[32] = ring_[warp];
    for (int task = (blockIdx.x / ng) * 8 + warp; task < ntask; task += (gridDim.x / ng) * 8) {
        // (the tasks of a warp are spread over the image: the same load for all)
        const int zb = task / npix, pix = task - zb * npix, c = zb * 32 + lane;
        const int o0 = offset[pix * nzb + zb], m = count[pix * nzb + zb];
        unsigned hi[ANR_MG], lo[ANR_MG];
#pragma unroll
        for (int i = 0; i < ANR_MG; i++) hi[i] = lo[i] = 0;
        int n = 0;                                          // deposits in hi and lo
        bool wide = false;                                  // sum is in use
        auto part = [&](int i) {
            return (unsigned long long)((long long)(int)(hi[i] - (unsigned)n * (unsigned)__float_as_int(ANF_HI)) *
                                            8388608 +
                                        (long long)(lo[i] - (unsigned)n * 0x4B000000u));
        };
        auto flush = [&]() {
#pragma unroll
            for (int i = 0; i < ANR_MG; i++) {
                sum[i][lane] = part(i) + (wide ? sum[i][lane] : 0ULL);
                hi[i] = lo[i] = 0;
            }
            wide = true;
            n = 0;
        };
        auto list = [&](int b0) { return lane < m - b0 ? __ldg(runs + o0 + b0 + lane) : make_int4(0, 0, 0, 0); };
        auto below = [&](const int4 &r) {
            return __ballot_sync(FULL, __int_as_float(r.w & 0xffff0000) * atop[r.w & 0xffff] < 0.5f * ANF_FIXMAX);
        };
        int4 q = list(0), qn = list(32);
        unsigned small = below(q);
        // the profiles of runs e and e + 1 in this lane's channel, on their way to the ring (0 outside a profile)
        auto fetch = [&](int e, const int4 &r) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int l = (e + u) & 31;
                const int s = __shfl_sync(FULL, r.x, l), kn = __shfl_sync(FULL, r.z, l), j = c - (kn & 0xffff);
                const bool in = (unsigned)j < ((unsigned)kn >> 16);
                const unsigned d = (unsigned)__cvta_generic_to_shared(&ring[(e + u) & (ANR_D - 1)][lane]);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d),
                             "l"(prof + (in ? (size_t)s * kw + j : 0)), "r"(in ? 4 : 0)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
#pragma unroll
        for (int e = 0; e < ANR_D - 2; e += 2) fetch(e, q);
        // (two runs a step: their parts join a sum in one three-operand addition; an odd last one is paired with an
        // empty run)
        for (int e = 0; e < m; e += 2) {
            const int l = e & 31, en = e + ANR_D - 2;
            if (l == 0 && e) {
                q = qn;
                qn = list(e + 32);
                small = below(q);
            }
            fetch(en, (en ^ e) & 32 ? qn : q);
            asm volatile("cp.async.wait_group %0;\n" ::"n"(ANR_D / 2 - 1) : "memory");
            const float b = ring[e & (ANR_D - 1)][lane], bb = ring[(e + 1) & (ANR_D - 1)][lane];
            const float w = __int_as_float(__shfl_sync(FULL, q.y, l));
            const float ww = __int_as_float(__shfl_sync(FULL, q.y, l + 1));
            const float4 *a4 = (const float4 *)(anr_amp + (__shfl_sync(FULL, q.w, l) & 0xffff) * ANR_MG);
            const float4 *aa4 = (const float4 *)(anr_amp + (__shfl_sync(FULL, q.w, l + 1) & 0xffff) * ANR_MG);
            if (((small >> l) & 3u) == 3u) {
                const unsigned long long b2 = f32x2(b, b), w2 = f32x2(w, w);
                const unsigned long long bb2 = f32x2(bb, bb), ww2 = f32x2(ww, ww);
#pragma unroll
                for (int i = 0; i < ANR_MG; i += 4) {
                    const float4 a = a4[i / 4], aa = aa4[i / 4];
                    unsigned long long t, q2, tt, qq;
                    fix_parts(f32x2_mul(f32x2_mul(b2, f32x2(a.x, a.y)), w2), t, q2);
                    fix_parts(f32x2_mul(f32x2_mul(bb2, f32x2(aa.x, aa.y)), ww2), tt, qq);
                    hi[i] += (unsigned)t + (unsigned)tt;
                    lo[i] += (unsigned)q2 + (unsigned)qq;
                    hi[i + 1] += (unsigned)(t >> 32) + (unsigned)(tt >> 32);
                    lo[i + 1] += (unsigned)(q2 >> 32) + (unsigned)(qq >> 32);
                    fix_parts(f32x2_mul(f32x2_mul(b2, f32x2(a.z, a.w)), w2), t, q2);
                    fix_parts(f32x2_mul(f32x2_mul(bb2, f32x2(aa.z, aa.w)), ww2), tt, qq);
                    hi[i + 2] += (unsigned)t + (unsigned)tt;
                    lo[i + 2] += (unsigned)q2 + (unsigned)qq;
                    hi[i + 3] += (unsigned)(t >> 32) + (unsigned)(tt >> 32);
                    lo[i + 3] += (unsigned)(q2 >> 32) + (unsigned)(qq >> 32);
                }
                n += 2;
                if (n == ANR_FLUSH) flush();
            } else {
                if (!wide) flush();
                for (int i = 0; i < ANR_MG; i++) {
                    sum[i][lane] += (unsigned long long)f32_to_ll(b * ((const float *)a4)[i] * w);
                    sum[i][lane] += (unsigned long long)f32_to_ll(bb * ((const float *)aa4)[i] * ww);
                }
            }
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (c >= nz) continue;
#pragma unroll
        for (int i = 0; i < ANR_MG; i++) {
            const int mi = grp * ANR_MG + i;
            if (mi < n3) {
                const int k = __ldg(klist + mi);
                const size_t at = (size_t)k * mstride + (size_t)pix * nz + c;
                model[at] = fix_to_f32((long long)(part(i) + (wide ? sum[i][lane] : 0ULL) + own[at]), mem[k].fix_exp);
            }
        }
    }
}

// ------------------------------------------------------------------------------ thin disks, by pixels
// A batch whose sub-rings all have one height (nzz = 1) and the float32 path. Each sample falls in one pixel, so the
// samples are listed by pixel (k_ant_bin, a scan, k_ant_list) and a warp takes a pixel with all its channels: it adds
// the deposits to a row of sums in shared memory that no other warp touches (64-bit fixed point: any order) and writes
// the pixel's float32 model. No memset, no 64-bit model in HBM, no atomics on sums, no conversion pass. The deposits are
// those of k_an_model_fast, integer for integer.
#define ANT_NT 256

// A sample as its pixel's warp deposits it: the line (velocity about vref in float-float, 1 / sig, amplitude in fixed-point
// units), the weight of its height and its channels k0 .. k0 + nk.
struct __align__(16) AntSample {
    float vrh, vrl, invf, amp, ws;
    unsigned short k0, nk;
    int pad[2];
};

// one thread per sample of the batch's segments: the record, its pixel (pixels of all members numbered from pix0[k];
// -1: nothing to deposit) and its rank among the pixel's samples (lanes of one pixel count once)
__global__ void __launch_bounds__(256) k_ant_bin(GridDev g, const AnSub *__restrict__ subs, int nsub,
                                                 const int *__restrict__ sbase, const int *__restrict__ ssub,
                                                 const double2 *__restrict__ cs, const float2 *__restrict__ csf,
                                                 const float4 *__restrict__ csff, const long long *__restrict__ astart,
                                                 const int4 *__restrict__ aseg, int nseg, long long ntot,
                                                 const int *__restrict__ pix0, const double *__restrict__ zq, const float *__restrict__ zqf,
                                                 const float *__restrict__ wqf, const MemberDev *__restrict__ mem,
                                                 AntSample *__restrict__ rec, int2 *__restrict__ where,
                                                 int *__restrict__ count) {
    const int lane = threadIdx.x & 31;
    const long long gs = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int pix = -1;
    AnSeg sg;
    if (an_seg(gs, astart, aseg, nseg, ntot, sbase, sg)) {
        const int s = (int)sg.s, ir = ssub[s];
        const AnSub &S = subs[(size_t)sg.src * nsub + ir];
        const float2 cf = csf[s];
        const bool rcd = cf.x >= 0.0f;                      // (the sign of the float32 table is the float64 test's)
        if (S.active && !(S.wzero & (rcd ? 1 : 2))) {
            const int kr = s - sbase[ir] >= S.naz ? 1 : 0;
            const PixF px = pix_setup(S, kr, cf, zqf + S.zq_off, 1);
            int g0, g1;
            sample_pixel(S, px, kr, cs + s, 1, 0.f, zq + S.zq_off, g.cdelt0, g.cdelt1, g0, g1);
            const MemberDev &M = mem[sg.k];
            g0 -= M.blo0;
            g1 -= M.blo1;
            if ((unsigned)g0 < (unsigned)M.bx && (unsigned)g1 < (unsigned)M.by) {
                ff v;
                const long long kc = fast_line_centre(S, g, csff[s], cs + s, v);
                long long a0 = kc - S.K, a1 = kc + S.K + 1;
                if (a0 < 0) a0 = 0;
                if (a1 > g.nz) a1 = g.nz;
                if (a1 > a0) {
                    pix = pix0[sg.k] + g1 * M.bx + g0;
                    const ff vr = ff_add(v, ff{-g.vrefh, -g.vrefl});
                    AntSample o;
                    o.vrh = vr.hi;
                    o.vrl = vr.lo;
                    o.invf = S.invf;
                    o.amp = (float)sg.sign * ldexpf(S.af * (rcd ? S.wrecf : S.wappf), M.fix_exp);
                    o.ws = wqf[S.zq_off];
                    o.k0 = (unsigned short)a0;
                    o.nk = (unsigned short)(a1 - a0);
                    o.pad[0] = o.pad[1] = 0;
                    rec[gs] = o;
                }
            }
        }
    }
    // consecutive samples often share a pixel: one atomic for each of the warp's pixels
    const unsigned same = __match_any_sync(FULL, pix);
    int r = 0;
    if (pix >= 0 && lane == __ffs(same) - 1) r = atomicAdd(count + pix, __popc(same));
    r = __shfl_sync(FULL, r, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1u));
    if (gs < ntot) where[gs] = make_int2(pix, r);
}

__global__ void k_ant_list(const int2 *__restrict__ where, long long ntot, const int *__restrict__ offset,
                           int *__restrict__ order) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntot) return;
    const int2 t = where[i];
    if (t.x >= 0) order[offset[t.x] + t.y] = (int)i;
}

__device__ __host__ inline int ant_pitch(int nz) { return (nz + 3) & ~1; }     // (sums of a warp: 16-byte rows)

// The pixels of the members [kfirst, kfirst + nk) (numbered pix0[kfirst] .. pix0[kfirst + nk)), a pixel a warp:
// persistent, so that the CDF table is read into shared memory once. 32 samples at a time are gathered a lane each; of
// a sample, a lane takes an edge of the line (its upper edge is the next lane's: 31 channels a step), always of a
// channel that is the lane's number modulo 32, so that no lane adds to another's sums; the 16-byte writes take four
// neighbouring sums a lane, behind a warp barrier. Bound by issue (about 90 instructions a step): 256 members of
// 256x256x192 7.3 ms (8.8 ms with 4-byte writes), where tiles of pixels with shared-memory atomics, the samples' edges
// laid end to end, took 8.9 ms. A pixel without samples, four in five, is only written. base64: member 0's sums in its
// box, written with base_out (by a launch of member 0 alone), else added to the members with mbase >= 0.
__global__ void __launch_bounds__(ANT_NT) k_ant_pixel(int nz, const int *__restrict__ pix0, int kfirst, int nk,
                                                      const int *__restrict__ offset, const int *__restrict__ count,
                                                      const int *__restrict__ order,
                                                      const AntSample *__restrict__ rec,
                                                      const float2 *__restrict__ vef, const float *__restrict__ cd2if,
                                                      const float *__restrict__ ptabf,
                                                      const MemberDev *__restrict__ mem, float *__restrict__ model,
                                                      double *__restrict__ model64, long long mstride,
                                                      long long *__restrict__ base64, int base_out,
                                                      const int *__restrict__ mbase) {
    // samples, (upper edge in float-float, factor) of the channels, sums of each warp, CDF
    extern __shared__ __align__(16) uint8_t ant_smem_[];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    AntSample *const rs = (AntSample *)ant_smem_ + w * 32;
    float4 *const chan = (float4 *)(ant_smem_ + nw * 32 * sizeof(AntSample));
    unsigned long long *const rows = (unsigned long long *)(chan + nz + 1), *const row = rows + (size_t)w * ant_pitch(nz);
    float *const tab = (float *)(rows + (size_t)nw * ant_pitch(nz));
    for (int i = tid; i < PHI_N; i += blockDim.x) tab[i] = ptabf[i];
    for (int i = tid; i <= nz; i += blockDim.x) {
        const float2 e = vef[i];
        chan[i] = make_float4(e.x, e.y, i < nz ? cd2if[i] : 0.0f, 0.0f);
    }
    for (int i = lane; i < nz; i += 32) row[i] = 0;
    __syncthreads();
    const int pend = pix0[kfirst + nk];
    const bool vec = (nz & 3) == 0 && (mstride & 3) == 0 && ((uintptr_t)model & 15) == 0;
    int k = kfirst;
    for (int t = pix0[kfirst] + blockIdx.x * nw + w; t < pend; t += gridDim.x * nw) {
        while (t >= pix0[k + 1]) k++;
        const int n = count[t], o0 = n ? offset[t] : 0;
        int c0 = nz, c1 = 0;                                // the channels with deposits
        for (int b0 = 0; b0 < n; b0 += 32) {
            const int m = min(32, n - b0);
            __syncwarp();                                   // (the samples before are done with)
            if (lane < m) rs[lane] = rec[order[o0 + b0 + lane]];
            __syncwarp();
            for (int i = 0; i < m; i++) {
                const AntSample q = rs[i];
                const int ka = q.k0, kb = ka + q.nk;
                c0 = min(c0, ka);
                c1 = max(c1, kb);
                for (int a = ka; a < kb; a += 31) {
                    const int c = a + ((lane - a) & 31), ce = min(c, kb);
                    const float4 ed = chan[ce];
                    const float f = phi_f32((__fsub_rn(ed.x, q.vrh) + __fsub_rn(ed.y, q.vrl)) * q.invf, tab);
                    const float fn = __shfl_sync(FULL, f, (lane + 1) & 31);
                    if (c < min(kb, a + 31)) {
                        const float x = fabsf(fn - f) * ed.z * q.amp * q.ws;
                        row[c] += fabsf(x) < ANF_FIXMAX ? f32_to_fix(x) : (unsigned long long)f32_to_ll(x);
                    }
                }
            }
        }
        __syncwarp();                                       // (a 16-byte write takes the sums of four lanes)
        const MemberDev &M = mem[k];
        const long long at = (long long)(t - pix0[k]) * nz;
        const long long *bas = !base_out && mbase[k] >= 0 ? base64 : nullptr;
        float *const out = model + (size_t)k * mstride + at;
        double *const out64 = model64 ? model64 + (size_t)k * mstride + at : nullptr;
        const int e = M.fix_exp;
        if (vec && !base_out && !bas && !out64) {           // (16-byte writes, four channels a lane)
            for (int c = 4 * lane; c < nz; c += 128) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (c < c1 && c + 4 > c0) {
                    ulonglong2 *const r = (ulonglong2 *)(row + c);
                    const ulonglong2 a = r[0], b = r[1];
                    r[0] = r[1] = make_ulonglong2(0ULL, 0ULL);
                    v = make_float4(fix_to_f32((long long)a.x, e), fix_to_f32((long long)a.y, e),
                                    fix_to_f32((long long)b.x, e), fix_to_f32((long long)b.y, e));
                }
                *(float4 *)(out + c) = v;
            }
            continue;
        }
        for (int c = lane; c < nz; c += 32) {
            unsigned long long q = 0;
            if (c >= c0 && c < c1) {
                q = row[c];
                row[c] = 0;
            }
            if (base_out) base64[at + c] = (long long)q;
            if (bas) q += (unsigned long long)bas[at + c];
            out[c] = q ? fix_to_f32((long long)q, e) : 0.0f;
            if (out64) out64[c] = __dmul_rn((double)(long long)q, ldexp(1.0, -e));
        }
    }
}

// Ring maps: maps64 (nr, by, bx) += fixed-point weights of the runs (bbarolo/galmod.py:518-529).
__global__ void __launch_bounds__(AN_WPB * 32) k_an_maps(GridDev g, const AnSub *__restrict__ subs, int nsub,
                                                         const int *__restrict__ sbase, const int *__restrict__ ssub,
                                                         const double2 *__restrict__ cs, long long nsamp,
                                                         const double *__restrict__ zq, const double *__restrict__ wq,
                                                         const long long *__restrict__ widx,
                                                         const double *__restrict__ wval, MemberDev M,
                                                         unsigned long long *__restrict__ maps64) {
    __shared__ AnWarp wsm[AN_WPB];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long gs = (long long)blockIdx.x * AN_WPB + w;
    if (gs >= nsamp) return;
    const AnSub *Sp;
    double caz, saz, R;
    if (!an_sample(gs, 0, nsub, subs, sbase, ssub, cs, Sp, caz, saz, R)) return;
    const AnSub &S = *Sp;
    const double wside = caz >= 0.0 ? S.wrec : S.wapp;
    if (wside == 0.0) return;
    AnWarp &W = wsm[w];
    const double fscale = ldexp(1.0, M.fix_exp);
    const double x = __dmul_rn(R, caz);
    const double yb = __dmul_rn(__dmul_rn(R, saz), S.cinc);
    const double xs = __dmul_rn(x, S.spa), xc = __dmul_rn(x, S.cpa);
    const size_t plane = (size_t)M.by * M.bx;
    auto emit = [&](int g0, int g1, double ws) {
        if (g0 < M.blo0 || g0 >= M.bhi0 || g1 < M.blo1 || g1 >= M.bhi1) return;
        if (lane < 2) {
            const long long r = widx[2 * S.sub + lane];
            if (r >= 0) {
                const double t = __dmul_rn(__dmul_rn(__dmul_rn(S.fluxsc, ws), wval[2 * S.sub + lane]), wside);
                const long long q = __double2ll_rn(__dmul_rn(t, fscale));
                if (q)
                    atomicAdd(maps64 + (size_t)r * plane + (size_t)(g1 - M.blo1) * M.bx + (size_t)(g0 - M.blo0),
                              (unsigned long long)q);
            }
        }
    };
    an_runs(S, zq + S.zq_off, wq + S.zq_off, g.cdelt0, g.cdelt1, xs, xc, yb, W.sgx, W.sgy, W.rg0, W.rg1, W.rws,
            emit);
}

// fixed point (units 2^-e of member k) -> float32 model and, optionally, float64 copy
// (mbase[k] >= 0: member k holds the difference from that member's sums, added modulo 2^64: the same box and unit)
__global__ void k_fix_to_model(const long long *__restrict__ in, const MemberDev *__restrict__ mem, long long mstride,
                               int nz, float *__restrict__ model, double *__restrict__ model64,
                               const int *__restrict__ mbase) {
    const int k = blockIdx.y;
    if (mbase && mbase[k] == -2) return;                    // (k_an_replay wrote it)
    const MemberDev &M = mem[k];
    const long long n = (long long)M.by * M.bx * nz;
    const int e = M.fix_exp;
    const long long *src = in + (size_t)k * mstride;
    const long long *bas = mbase && mbase[k] >= 0 ? in + (size_t)mbase[k] * mstride : nullptr;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        long long q = src[i];
        if (bas) q = (long long)((unsigned long long)q + (unsigned long long)bas[i]);
        model[(size_t)k * mstride + i] = fix_to_f32(q, e);
        if (model64) model64[(size_t)k * mstride + i] = __dmul_rn((double)q, ldexp(1.0, -e));
    }
}

}  // namespace

size_t an_smem_bytes(int nz, int nlines) { return (size_t)AN_WPB * nlines * (nz + 2) * sizeof(double); }

void launch_an_model(cudaStream_t s, const GridDev &g, const AnSub *subs, int nsub, const int *sbase, const int *ssub,
                     const double *cs, const float *csf, const long long *astart, const int *aseg, int nseg,
                     long long ntot, const double *zq, const double *wq, const float *zqf, const double *vedges, const double *cd2i, const double *ptab,
                     const MemberDev *mem, long long *out64, long long mstride, int skip_fast) {
    const long long nw = ntot;
    if (nw == 0 || nseg == 0) return;
    const size_t smem = an_smem_bytes(g.nz, g.nlines);
    allow_smem((const void *)k_an_model, smem);
    k_an_model<<<(unsigned)((nw + AN_WPB - 1) / AN_WPB), AN_WPB * 32, smem, s>>>(
        g, subs, nsub, sbase, ssub, (const double2 *)cs, (const float2 *)csf, astart, (const int4 *)aseg, nseg, ntot, zq,
        wq, zqf, vedges, cd2i, ptab, mem, (unsigned long long *)out64, mstride, skip_fast);
}

void launch_an_model_fast(cudaStream_t s, const GridDev &g, const AnSub *subs, int nsub, const int *sbase,
                          const int *ssub, const double *cs, const float *csf, const float *csff,
                          const long long *astart, const int *aseg, int nseg, long long ntot,
                          const double *zq, const float *zqf, const float *wqf, const float *vef, const float *cd2if,
                          const float *ptabf, const MemberDev *mem, long long *out64, long long mstride) {
    if (ntot == 0 || nseg == 0) return;
    const long long per = 32 * ANF_WPB;
    const size_t smem = ANF_WPB * (32 * sizeof(AnfSample) + ANF_RUNS * sizeof(int2)) + (PHI_N + (size_t)ANF_WPB * g.nz) * 4;
    allow_smem((const void *)k_an_model_fast, smem);
    k_an_model_fast<<<(unsigned)((ntot + per - 1) / per), ANF_WPB * 32, smem, s>>>(
        g, subs, nsub, sbase, ssub, (const double2 *)cs, (const float2 *)csf, (const float4 *)csff, astart,
        (const int4 *)aseg, nseg, ntot, zq, zqf, wqf, (const float2 *)vef, cd2if, ptabf, mem,
        (unsigned long long *)out64, mstride);
}

void launch_an_records(cudaStream_t s, const GridDev &g, const AnSub *subs, const int *sbase, const int *ssub,
                       const double *cs, const float *csf, const float *csff, long long ns,
                       const unsigned long long *act, const double *zq, const float *zqf, const float *wqf,
                       const float *vef, const float *cd2if, const float *ptabf, const MemberDev *mem, int nlist,
                       int *count, int *scan, void *runs, float *prof, int kw) {
    const unsigned grid = (unsigned)((ns + 32 * ANF_WPB - 1) / (32 * ANF_WPB));
    int *const offset = count + nlist + 1, *const cursor = offset + nlist + 1;
    cudaMemsetAsync(count, 0, sizeof(int) * (nlist + 1), s);
    if (!grid) return;
    k_an_records<false><<<grid, ANF_WPB * 32, 0, s>>>(g, subs, sbase, ssub, (const double2 *)cs, (const float2 *)csf,
                                                      (const float4 *)csff, ns, act, zq, zqf, wqf, (const float2 *)vef,
                                                      cd2if, ptabf, mem, count, nullptr, nullptr, kw);
    launch_scan_tiles(s, count, offset, cursor, nlist, scan);
    k_an_records<true><<<grid, ANF_WPB * 32, 0, s>>>(g, subs, sbase, ssub, (const double2 *)cs, (const float2 *)csf,
                                                     (const float4 *)csff, ns, act, zq, zqf, wqf, (const float2 *)vef,
                                                     cd2if, ptabf, mem, cursor, (AnRun *)runs, prof, kw);
}

int an_replay_groups(int n3) { return (n3 + ANR_MG - 1) / ANR_MG; }
bool an_replay_fits(int nsub) { return nsub <= 640; }

void launch_an_replay(cudaStream_t s, const GridDev &g, const AnSub *subs, int nsub, const MemberDev *mem, int npix,
                      const int *klist, int n3, const unsigned long long *chg, int nchw, const int *count,
                      const void *runs, const float *prof, int kw, float *amp, const long long *own, long long mstride,
                      float *model) {
    const int ng = an_replay_groups(n3), nzb = (g.nz + 31) / 32, ntask = npix * nzb;
    const long long na = 2LL * nsub * ng * ANR_MG;
    if (!na || !ntask) return;
    float *const top = amp + na;
    k_an_amps<<<(unsigned)((na + 255) / 256), 256, 0, s>>>(subs, nsub, mem, klist, n3, ng, chg, nchw, amp, top);
    const size_t smem = (size_t)2 * nsub * (ANR_MG + 1) * sizeof(float);
    allow_smem((const void *)k_an_replay, smem);
    const int nc = std::max(1, std::min(sm_count() * resident_ctas((const void *)k_an_replay, 256, smem) / ng,
                                        (ntask + 7) / 8));
    k_an_replay<<<nc * ng, 256, smem, s>>>(g.nz, ng, nzb, npix, ntask, 2 * nsub, count + ntask + 1, count,
                                           (const int4 *)runs, prof, kw, amp, top, klist, n3, mem, (const unsigned long long *)own, mstride,
                                           model);
}

// shared memory of k_ant_pixel with nw warps a CTA; the warps that fit (8, or fewer for many channels; 0: none)
static size_t ant_smem(int nz, int nw) {
    return nw * (32 * sizeof(AntSample) + (size_t)ant_pitch(nz) * 8) + ((size_t)nz + 1) * 16 + PHI_N * 4;
}
int ant_warps(int nz) {
    if (nz >= 65536) return 0;
    for (int nw = ANT_NT / 32; nw > 0; nw >>= 1)
        if (ant_smem(nz, nw) <= AN_SMEM_MAX) return nw;
    return 0;
}

void launch_ant_bin(cudaStream_t s, const GridDev &g, const AnSub *subs, int nsub, const int *sbase, const int *ssub,
                    const double *cs, const float *csf, const float *csff, const long long *astart, const int *aseg,
                    int nseg, long long ntot, const int *pix0, const double *zq, const float *zqf,
                    const float *wqf, const MemberDev *mem, void *rec, int *where, int *count) {
    if (ntot == 0 || nseg == 0) return;
    k_ant_bin<<<(unsigned)((ntot + 255) / 256), 256, 0, s>>>(
        g, subs, nsub, sbase, ssub, (const double2 *)cs, (const float2 *)csf, (const float4 *)csff, astart,
        (const int4 *)aseg, nseg, ntot, pix0, zq, zqf, wqf, mem, (AntSample *)rec, (int2 *)where, count);
}

void launch_ant_list(cudaStream_t s, const int *where, long long ntot, const int *offset, int *order) {
    if (ntot == 0) return;
    k_ant_list<<<(unsigned)((ntot + 255) / 256), 256, 0, s>>>((const int2 *)where, ntot, offset, order);
}

void launch_ant_pixel(cudaStream_t s, int nz, const int *pix0, int kfirst, int nk, int npix, const int *offset,
                      const int *count, const int *order, const void *rec, const float *vef, const float *cd2if,
                      const float *ptabf, const MemberDev *mem, float *model, double *model64, long long mstride,
                      long long *base64, int base_out, const int *mbase) {
    const int nw = ant_warps(nz);
    if (nk <= 0 || npix <= 0 || !nw) return;
    const size_t smem = ant_smem(nz, nw);
    allow_smem((const void *)k_ant_pixel, smem);
    const int fill = sm_count() * resident_ctas((const void *)k_ant_pixel, 32 * nw, smem);
    k_ant_pixel<<<std::min((npix + nw - 1) / nw, fill), 32 * nw, smem, s>>>(
        nz, pix0, kfirst, nk, offset, count, order, (const AntSample *)rec, (const float2 *)vef, cd2if, ptabf, mem,
        model, model64, mstride, base64, base_out, mbase);
}

void launch_an_maps(cudaStream_t s, const GridDev &g, const AnSub *subs, int nsub, const int *sbase, const int *ssub,
                    const double *cs, long long nsamp, const double *zq, const double *wq, const long long *widx,
                    const double *wval, const MemberDev &M, long long *maps64) {
    if (nsamp == 0) return;
    k_an_maps<<<(unsigned)((nsamp + AN_WPB - 1) / AN_WPB), AN_WPB * 32, 0, s>>>(
        g, subs, nsub, sbase, ssub, (const double2 *)cs, nsamp, zq, wq, widx, wval, M, (unsigned long long *)maps64);
}

void launch_fix_to_model(cudaStream_t s, const long long *in, const MemberDev *mem, int nb, long long mstride, int nz,
                         float *model, double *model64, const int *mbase) {
    if (nb == 0) return;
    dim3 grid(256, nb);
    k_fix_to_model<<<grid, 256, 0, s>>>(in, mem, mstride, nz, model, model64, mbase);
}
