// GALWIND WTYPE 1 on the device: the Monte-Carlo clouds of spherical shells of a bi-cone (the reference's
// _galmod_wind, bbarolo/galmod.py:539-590).
//
// The reference draws a cloud's radius, azimuth and polar angle (a word of the stream each) and its velocity deviates
// (ziggurat normals: one word each but for about 3%), so where a cloud's words lie depends on every draw before it.
// That chain is followed on the device (k_ws_*) when all the shells have the same number of velocity samples:
//   gen     the words: segments of WS_SEG steps, each from the stream's state moved there by its linear map (a product
//           of precomputed powers), with a bit for every word that would leave the ziggurat's one-word path;
//   fails   those words listed in order, and for each how many further words a deviate starting there takes, and its value;
//   spec    per block of words and per possible place in a cloud's cycle of draws at its start: the words it takes
//           beyond one a draw (a walk over the block's failing words);
//   chain   the blocks' true starts by look-up, groups of blocks first;
//   place   every block again from its true start: the first word of each cloud;
//   clouds  a thread a cloud: its pixel and the channel of every velocity sample.
// 2.2 M clouds of 20 samples (45 M words) in 16 chunks: 43 ms with the streams parsed on 16 host threads,
// 2.6 ms followed here (2.1 of it on the device, 0.9 the clouds: float64 sines and positions).
// Otherwise (other counts, a handful of draws) the host parses the stream into the clouds and their deviates
// (bbh_wind_clouds) and k_wind_mc places them.
//
// A cloud is placed with the reference's float64 operations in its order, no contraction, and deposited in 64-bit fixed
// point (units 2^(E-62), 2^E above the total flux of the clouds: exact sums, independent of their order). From the host
// parse its pixel and channels are the reference's. On the device sin, cos, log and exp are within two ulps of the C
// library's: where that could move a pixel, a channel or a deviate's rejection, the launch says so (WS_NEAR) and the
// host parse makes the model, so that the same holds (about one model of 2.2 M clouds in ten thousand).
#include <cuda_runtime.h>
#include <stdint.h>

#include "devmath.cuh"
#include "kernels.h"

namespace {

__global__ void __launch_bounds__(256) k_wind_mc(const WindShell *__restrict__ shells, const int *__restrict__ shell,
                                                 const double *__restrict__ geo, const long long *__restrict__ nbase,
                                                 const long long *__restrict__ sbase, const int *__restrict__ hz,
                                                 const double *__restrict__ slow, const ZigDev *__restrict__ zig,
                                                 long long ncloud, GridDev g,
                                                 const double *__restrict__ cd2i, int blo0, int blo1, int bhi0,
                                                 int bhi1, double scale, unsigned long long *__restrict__ acc) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncloud) return;
    const WindShell s = shells[shell[i]];
    const double *c = geo + 5 * (size_t)i;
    const double rad = c[0], caz = c[1], saz = c[2], sphi = c[3], cphi = c[4];
    // bbarolo/galmod.py:568-575
    const double R = __dmul_rn(rad, sphi), z = __dmul_rn(rad, cphi);
    const double x = __dmul_rn(R, caz);
    const double y = __dsub_rn(__dmul_rn(__dmul_rn(R, saz), s.cinc), __dmul_rn(z, s.sinc));
    const long long g0 =
        lround_ref(__dadd_rn(s.xpos, __ddiv_rn(__dsub_rn(__dmul_rn(x, s.spa), __dmul_rn(y, s.cpa)), g.cdelt0)));
    const long long g1 =
        lround_ref(__dadd_rn(s.ypos, __ddiv_rn(__dadd_rn(__dmul_rn(x, s.cpa), __dmul_rn(y, s.spa)), g.cdelt1)));
    if (g0 < blo0 || g0 >= bhi0 || g1 < blo1 || g1 >= bhi1) return;
    // bbarolo/galmod.py:581-589
    const double geom = __dadd_rn(__dmul_rn(cphi, s.cinc), __dmul_rn(__dmul_rn(sphi, saz), s.sinc));
    const double vs = __dadd_rn(__dadd_rn(s.vsys, __dmul_rn(s.vsph, geom)), __dmul_rn(__dmul_rn(s.vrot, caz), s.sinc));
    unsigned long long *o = acc + ((size_t)(g1 - blo1) * (bhi0 - blo0) + (size_t)(g0 - blo0)) * g.nz;
    const int *h = hz + nbase[i];
    long long js = sbase[i];
    for (int iv = 0; iv < s.nvr; iv++) {
        // the deviate: from its first word on the ziggurat's one-word path (the reference's product), else recorded
        const int hv = h[iv];
        const unsigned ah = hv < 0 ? 0u - (unsigned)hv : (unsigned)hv;
        const double n = ah < zig->kn[hv & 127] ? __dmul_rn((double)hv, zig->wn[hv & 127]) : slow[js++];
        const double v = __dadd_rn(vs, __dmul_rn(n, s.vdisp));
        for (int nl = 0; nl < g.nlines; nl++) {
            const long long k = lround_ref(velgrid_exact(v, g, nl));
            if (k < 0 || k >= g.nz) continue;
            const double val = __dmul_rn(__dmul_rn(g.relint[nl], s.fluxsc), cd2i[k]);
            atomicAdd(o + k, (unsigned long long)__double2ll_rn(val * scale));
        }
    }
}

// ------------------------------------------------------------------------------------- the stream on the device
__device__ __forceinline__ bool ws_fast(unsigned long long w, const unsigned *kn, int &hv) {
    hv = (int)((unsigned)(w >> 32) - 0x80000000u);
    const unsigned ah = hv < 0 ? 0u - (unsigned)hv : (unsigned)hv;
    return ah < kn[hv & 127];
}

__device__ __forceinline__ double ws_uniform(unsigned long long w) {
    return __dmul_rn((double)(w >> 11), 1.0 / 9007199254740992.0);
}

// the job of item i by the jobs' first items (field of WindJob)
template <class F>
__device__ __forceinline__ int ws_job(const WindJob *jobs, int njob, long long i, F first) {
    int lo = 0, hi = njob - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (first(jobs[mid]) <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// a warp: 32 segments, a lane each, 32 words at a time turned over in shared memory to be written in order
__global__ void __launch_bounds__(128) k_ws_gen(const WindJob *__restrict__ jobs, int njob, int nseg,
                                                const ulonglong2 *__restrict__ jump, const ZigDev *__restrict__ zig,
                                                unsigned long long *__restrict__ words, unsigned *__restrict__ masks,
                                                int *__restrict__ nfail) {
    __shared__ unsigned long long tile[4][32][33];
    __shared__ unsigned kn[128];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    kn[threadIdx.x] = zig->kn[threadIdx.x];
    __syncthreads();
    const int seg0 = (blockIdx.x * 4 + w) * 32, seg = min(seg0 + lane, nseg - 1);
    if (seg0 >= nseg) return;
    const WindJob &J = jobs[ws_job(jobs, njob, seg, [](const WindJob &j) { return (long long)j.seg0; })];
    unsigned long long s0 = J.s0, s1 = J.s1;
    const unsigned at = (unsigned)(J.segbase + (seg - J.seg0));
    const int top = 32 - __clz((int)__reduce_max_sync(0xffffffffu, at));
    for (int b = 0; b < top; b++) {
        unsigned long long a0 = 0, a1 = 0;
        const ulonglong2 *m = jump + 128 * b;
        for (int i = 0; i < 64; i++) {
            const ulonglong2 c0 = __ldg(m + i), c1 = __ldg(m + 64 + i);
            const unsigned long long k0 = 0ULL - ((s0 >> i) & 1), k1 = 0ULL - ((s1 >> i) & 1);
            a0 ^= (c0.x & k0) ^ (c1.x & k1);
            a1 ^= (c0.y & k0) ^ (c1.y & k1);
        }
        if ((at >> b) & 1) {
            s0 = a0;
            s1 = a1;
        }
    }
    int cnt = 0;
    for (int t = 0; t < WS_SEG / 32; t++) {
#pragma unroll 8
        for (int j = 0; j < 32; j++) {
            tile[w][lane][j] = s0 + s1;                     // xoroshiro128+
            s1 ^= s0;
            s0 = ((s0 << 24) | (s0 >> 40)) ^ s1 ^ (s1 << 16);
            s1 = (s1 << 37) | (s1 >> 27);
        }
        __syncwarp();
        unsigned mine = 0;
        for (int r = 0; r < 32 && seg0 + r < nseg; r++) {
            const unsigned long long v = tile[w][r][lane];
            int hv;
            const unsigned m = __ballot_sync(0xffffffffu, !ws_fast(v, kn, hv));
            words[(size_t)(seg0 + r) * WS_SEG + t * 32 + lane] = v;
            if (lane == r) mine = m;
        }
        if (seg0 + lane < nseg) masks[(size_t)(seg0 + lane) * (WS_SEG / 32) + t] = mine;
        cnt += __popc(mine);
        __syncwarp();
    }
    if (seg0 + lane < nseg) nfail[seg0 + lane] = cnt;
}

// v within 2^-20 of the middle between two integers (|v| < 2^31: one addition leaves 20 bits of the fraction)
__device__ __forceinline__ bool ws_close(double v) {
    return ((unsigned)__double2loint(__dadd_rn(v, 6442450944.0)) & 0xfffffu) - 0x7ffffu <= 2u;
}
// ... within tol, for which sin and cos 3.4e-16 off the C library's are enough: they move a cloud of radius rad by less
// than 5e-15 rad
__device__ __noinline__ bool ws_near(double v, double pos, double rad, double cdelt) {
    return fabs(__dsub_rn(__dsub_rn(v, floor(v)), 0.5)) < 1e-14 * (fabs(pos) + 4.0 * rad / fabs(cdelt));
}

// the positions of the failing words, in order: a thread a mask
__global__ void k_ws_list(const unsigned *__restrict__ masks, int nmask, const int *__restrict__ foff,
                          unsigned *__restrict__ fpos, int cap, int *__restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nmask) return;
    const int seg = i / (WS_SEG / 32), t = i % (WS_SEG / 32);
    int o = foff[seg];
    for (int q = 0; q < t; q++) o += __popc(masks[seg * (WS_SEG / 32) + q]);
    for (unsigned m = masks[i]; m; m &= m - 1, o++) {
        if (o < cap) fpos[o] = (unsigned)i * 32 + __ffs(m) - 1;
        else atomicOr(err, WS_LOST);
    }
}

// a deviate starting at each failing word (bbarolo/_rng.py:65-100): the further words it takes, its value
__global__ void k_ws_slow(const unsigned *__restrict__ fpos, const int *__restrict__ foff, int nseg,
                          const int *__restrict__ nfail, int cap, const unsigned long long *__restrict__ words,
                          unsigned nword, const ZigDev *__restrict__ zig, const double *__restrict__ fn,
                          unsigned char *__restrict__ fext, double *__restrict__ fval, int *__restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = min(cap, foff[nseg - 1] + nfail[nseg - 1]);
    if (i >= n) return;
    const unsigned p = fpos[i];
    unsigned q = p;
    double val = 0.0;
    const unsigned end = min(nword, p + 200u);              // (a deviate beyond 200 words does not occur)
    auto next = [&]() { return q < end ? words[q++] : (q++, 0ULL); };
    // (a < b of values that may each be a few ulps off)
    bool near = false;
    auto less = [&](double a, double b) {
        near |= fabs(__dsub_rn(a, b)) <= 1e-14 * fabs(b);
        return a < b;
    };
    for (;;) {
        int hv;
        const bool fast = ws_fast(next(), zig->kn, hv);
        const int iz = hv & 127;
        const double x = __dmul_rn((double)hv, zig->wn[iz]);
        val = x;
        if (fast || q > end) break;
        if (iz == 0) {
            double xx, yy;
            do {
                xx = __dmul_rn(-log(__dsub_rn(1.0, ws_uniform(next()))), 0.2904764);
                yy = -log(__dsub_rn(1.0, ws_uniform(next())));
            } while (less(__dadd_rn(yy, yy), __dmul_rn(xx, xx)) && q <= end);
            val = hv > 0 ? __dadd_rn(3.442620, xx) : __dsub_rn(-3.442620, xx);
            break;
        }
        const double f = __dadd_rn(fn[iz], __dmul_rn(ws_uniform(next()), __dsub_rn(fn[iz - 1], fn[iz])));
        if (less(f, exp(__dmul_rn(__dmul_rn(-.5, x), x)))) break;
    }
    fext[i] = (unsigned char)min(q - p - 1, 255u);
    fval[i] = val;
    // (the last words of the launch cannot be resolved; they are guard words, which no cloud that is placed reads)
    if (q > end && end != nword) atomicOr(err, WS_LOST);
    if (near && q <= end) atomicOr(err, WS_NEAR);
}

// per (block, place at its first word): the words beyond one a draw, and by how many words the last deviate runs over
// the block's end (upper half)
__global__ void k_ws_spec(const WindJob *__restrict__ jobs, int njob, int nblk, int M, const int *__restrict__ foff,
                          const unsigned *__restrict__ fpos, const unsigned char *__restrict__ fext, int cap,
                          unsigned *__restrict__ spec) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nblk * M) return;
    const int b = (int)(i / M);
    int c = (int)(i - (long long)b * M);                    // (place at the block's start, less the extra words, mod M)
    const WindJob &J = jobs[ws_job(jobs, njob, b, [](const WindJob &j) { return (long long)j.blk0; })];
    const int seg = J.seg0 + (b - J.blk0) * WS_BLK;
    const unsigned pb = (unsigned)seg * WS_SEG, pe = pb + WS_BLK * WS_SEG;
    unsigned pmin = pb;
    int extra = 0;
    for (int f = foff[seg], f1 = min(cap, foff[seg + WS_BLK]); f < f1; f++) {
        const unsigned p = fpos[f];
        if (p < pmin || (c + (p - pb)) % (unsigned)M < 3u) continue;
        const int e = fext[f];
        extra += e;
        c -= e % M;
        if (c < 0) c += M;
        pmin = p + 1 + e;
    }
    spec[i] = (unsigned)extra | ((pmin > pe ? pmin - pe : 0u) << 16);
}

// the start of the block after block b of job J, entered at s: looked up, or, past its first word, walked
__device__ __forceinline__ void ws_step(const WindJob &J, int b, int M, const int *foff, const unsigned *fpos,
                                        const unsigned char *fext, int cap, const unsigned *spec, WsStart &s) {
    const int B = WS_BLK * WS_SEG;
    int extra = 0, over = 0;
    if (s.skip == 0) {
        const unsigned v = spec[(size_t)(J.blk0 + b) * M + s.slot];
        extra = v & 0xffff;
        over = v >> 16;
    } else {
        const int seg = J.seg0 + b * WS_BLK;
        const unsigned p0 = (unsigned)seg * WS_SEG + s.skip, pe = (unsigned)seg * WS_SEG + B;
        unsigned pmin = p0;
        int c = s.slot;
        for (int f = foff[seg], f1 = min(cap, foff[seg + WS_BLK]); f < f1; f++) {
            const unsigned p = fpos[f];
            if (p < pmin || (c + (p - p0)) % (unsigned)M < 3u) continue;
            const int e = fext[f];
            extra += e;
            c -= e % M;
            if (c < 0) c += M;
            pmin = p + 1 + e;
        }
        over = pmin > pe ? (int)(pmin - pe) : 0;
    }
    const int draws = B + over - s.skip - extra;
    s.draw += draws;
    s.slot = (int)((unsigned)(s.slot + draws) % (unsigned)M);
    s.skip = over;
}

// The blocks one after another would be a chain of thousands of look-ups (1.3 ms for 690 blocks a chunk): groups of
// WS_GRP blocks are followed from every place at their first word side by side (k_ws_group), the chain goes over the
// groups (k_ws_chain), then every group fills in its blocks (k_ws_expand). group: (WsStart of the next group, draws
// counted from the group's start) per (group, place).
__global__ void k_ws_group(const WindJob *__restrict__ jobs, int njob, int ngrp, int M, const int *__restrict__ foff,
                           const unsigned *__restrict__ fpos, const unsigned char *__restrict__ fext, int cap,
                           const unsigned *__restrict__ spec, WsStart *__restrict__ group) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)ngrp * M) return;
    const int gr = (int)(i / M);
    const WindJob &J = jobs[ws_job(jobs, njob, gr, [](const WindJob &j) { return (long long)j.grp0; })];
    WsStart s{0, (int)(i - (long long)gr * M), 0};
    const int b0 = (gr - J.grp0) * WS_GRP, b1 = min(J.nblk, b0 + WS_GRP);
    for (int b = b0; b < b1; b++) ws_step(J, b, M, foff, fpos, fext, cap, spec, s);
    group[i] = s;
}

__global__ void k_ws_chain(const WindJob *__restrict__ jobs, int njob, int M, const int *__restrict__ foff,
                           const unsigned *__restrict__ fpos, const unsigned char *__restrict__ fext, int cap,
                           const unsigned *__restrict__ spec, const WsStart *__restrict__ group,
                           WsStart *__restrict__ gstart, WsStart *__restrict__ ends) {
    if (threadIdx.x) return;
    const WindJob &J = jobs[blockIdx.x];
    WsStart s = J.start;
    for (int b0 = 0, gr = J.grp0; b0 < J.nblk; b0 += WS_GRP, gr++) {
        gstart[gr] = s;
        if (s.skip == 0) {
            const WsStart t = group[(size_t)gr * M + s.slot];
            s.draw += t.draw;
            s.slot = t.slot;
            s.skip = t.skip;
        } else {
            for (int b = b0; b < min(J.nblk, b0 + WS_GRP); b++) ws_step(J, b, M, foff, fpos, fext, cap, spec, s);
        }
    }
    ends[blockIdx.x] = s;
}

__global__ void k_ws_expand(const WindJob *__restrict__ jobs, int njob, int ngrp, int M, const int *__restrict__ foff,
                            const unsigned *__restrict__ fpos, const unsigned char *__restrict__ fext, int cap,
                            const unsigned *__restrict__ spec, const WsStart *__restrict__ gstart,
                            WsStart *__restrict__ start) {
    const int gr = blockIdx.x * blockDim.x + threadIdx.x;
    if (gr >= ngrp) return;
    const WindJob &J = jobs[ws_job(jobs, njob, gr, [](const WindJob &j) { return (long long)j.grp0; })];
    WsStart s = gstart[gr];
    const int b0 = (gr - J.grp0) * WS_GRP, b1 = min(J.nblk, b0 + WS_GRP);
    for (int b = b0; b < b1; b++) {
        start[J.blk0 + b] = s;
        ws_step(J, b, M, foff, fpos, fext, cap, spec, s);
    }
}

// a thread per block: the first word and the first failing word of every cloud that starts in it
__global__ void k_ws_place(const WindJob *__restrict__ jobs, int njob, int nblk, int M, const int *__restrict__ foff,
                           const unsigned *__restrict__ fpos, const unsigned char *__restrict__ fext, int cap,
                           const WsStart *__restrict__ start, uint2 *__restrict__ cloud) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nblk) return;
    const WindJob &J = jobs[ws_job(jobs, njob, b, [](const WindJob &j) { return (long long)j.blk0; })];
    const int seg = J.seg0 + (b - J.blk0) * WS_BLK;
    const WsStart s = start[b];
    const unsigned pb = (unsigned)seg * WS_SEG, pe = pb + WS_BLK * WS_SEG;
    unsigned p = pb + s.skip, pmin = p, pc = p - s.slot;    // (pc: the first word of the cloud in hand, less its extras)
    unsigned pn = s.slot ? p + (M - s.slot) : p;            // the next cloud's first word
    long long k = (s.draw + M - 1) / M;
    for (int f = foff[seg], f1 = min(cap, foff[seg + WS_BLK]);;) {
        for (; f < f1; f++) {
            const unsigned q = fpos[f];
            if (q >= pn) break;
            if (q < pmin || q < p || q - pc < 3u) continue;
            const int e = fext[f];
            pn += e;
            pc += e;
            pmin = q + 1 + e;
        }
        if (pn >= pe || k - J.k0 >= J.ncl) return;
        cloud[J.cl0 + (k - J.k0)] = make_uint2(pn, f);
        k++;
        p = pmin = pc = pn;
        pn += M;
    }
}

// the deposit of a velocity sample per (shell, line, channel), in fixed point
__global__ void k_ws_flux(const WindShell *__restrict__ shells, int nshell, GridDev g, const double *__restrict__ cd2i,
                          double scale, long long *__restrict__ fix) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)nshell * g.nlines * g.nz) return;
    const int k = (int)(i % g.nz), nl = (int)(i / g.nz % g.nlines), sh = (int)(i / g.nz / g.nlines);
    fix[i] = __double2ll_rn(__dmul_rn(__dmul_rn(__dmul_rn(g.relint[nl], shells[sh].fluxsc), cd2i[k]), scale));
}

// A thread a cloud. The channel of a sample in float-float (the float64 pipe runs at 1/64 of the float32 rate here)
// where the channel map is linear: within 1e-6 of a channel boundary, and for further lines, the reference's float64
// operations. Four CTAs an SM: at 68 registers a thread, three, the model of 2.2 M clouds took 2.29 ms for 2.22.
__global__ void __launch_bounds__(256, 4) k_ws_clouds(const WindJob *__restrict__ jobs, int njob, long long ncl, int M,
                                                   const WsStart *__restrict__ ends,
                                                   const uint2 *__restrict__ cloud,
                                                   const unsigned long long *__restrict__ words,
                                                   const unsigned *__restrict__ fpos,
                                                   const unsigned char *__restrict__ fext,
                                                   const double *__restrict__ fval, const ZigDev *__restrict__ zig,
                                                   const WindShell *__restrict__ shells,
                                                   const WindCloudLaw *__restrict__ law,
                                                   const long long *__restrict__ sfirst, unsigned nword, int cap,
                                                   int *__restrict__ err, GridDev g, int blo0, int blo1,
                                                   int bhi0, int bhi1, const long long *__restrict__ fix,
                                                   unsigned long long *__restrict__ acc) {
    __shared__ unsigned kn[128];
    __shared__ float2 wnf[128];
    if (threadIdx.x < 128) {
        kn[threadIdx.x] = zig->kn[threadIdx.x];
        const ff t = ff_of(zig->wn[threadIdx.x]);
        wnf[threadIdx.x] = make_float2(t.hi, t.lo);
    }
    __syncthreads();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncl) return;
    const int jb = ws_job(jobs, njob, i, [](const WindJob &j) { return j.cl0; });
    const WindJob &J = jobs[jb];
    const long long k = J.k0 + (i - J.cl0);
    if (i - J.cl0 >= J.ncl || k * M >= ends[jb].draw) return;
    int lo = J.shell0, hi = J.shell0 + J.nshell - 1;        // its shell (sfirst: first cloud in the chunk)
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (sfirst[mid] <= k) lo = mid;
        else hi = mid - 1;
    }
    const WindShell &s = shells[lo];
    const WindCloudLaw L = law[lo];
    const uint2 at = cloud[i];
    const unsigned long long *w = words + at.x;
    // bbarolo/galmod.py:567-575
    const double pi = 3.14159265358979323846;
    auto sym = [](unsigned long long v) { return fabs(__dsub_rn(__dmul_rn(2.0, ws_uniform(v)), 1.0)); };
    const double rad = __dsqrt_rn(__dadd_rn(L.r2, __dmul_rn(L.rc, sym(w[0]))));
    const double az = __dmul_rn(2 * pi, sym(w[1]));
    double ph = __dmul_rn(L.open, sym(w[2]));
    if ((k - sfirst[lo]) % 2 == 0) ph = __dsub_rn(pi, ph);
    double saz, caz, sphi, cphi;
    sincos(az, &saz, &caz);
    sincos(ph, &sphi, &cphi);
    const double R = __dmul_rn(rad, sphi), z = __dmul_rn(rad, cphi);
    const double x = __dmul_rn(R, caz);
    const double y = __dsub_rn(__dmul_rn(__dmul_rn(R, saz), s.cinc), __dmul_rn(z, s.sinc));
    const double px = __dadd_rn(s.xpos, __ddiv_rn(__dsub_rn(__dmul_rn(x, s.spa), __dmul_rn(y, s.cpa)), g.cdelt0));
    const double py = __dadd_rn(s.ypos, __ddiv_rn(__dadd_rn(__dmul_rn(x, s.cpa), __dmul_rn(y, s.spa)), g.cdelt1));
    const long long g0 = lround_ref(px), g1 = lround_ref(py);
    if ((ws_close(px) && ws_near(px, s.xpos, rad, g.cdelt0)) || (ws_close(py) && ws_near(py, s.ypos, rad, g.cdelt1)))
        atomicOr(err, WS_NEAR);
    if (g0 < blo0 || g0 >= bhi0 || g1 < blo1 || g1 >= bhi1) return;
    // bbarolo/galmod.py:581-589
    const double geom = __dadd_rn(__dmul_rn(cphi, s.cinc), __dmul_rn(__dmul_rn(sphi, saz), s.sinc));
    const double vs = __dadd_rn(__dadd_rn(s.vsys, __dmul_rn(s.vsph, geom)), __dmul_rn(__dmul_rn(s.vrot, caz), s.sinc));
    unsigned long long *o = acc + ((size_t)(g1 - blo1) * (bhi0 - blo0) + (size_t)(g0 - blo0)) * g.nz;
    const long long *fx = fix + (size_t)lo * g.nlines * g.nz;
    const ff chw = ff_mul(ff_of(s.vdisp), ff{g.ia0h, g.ia0l});
    const ff ch0 = ff_add(ff_mul(ff_of(vs), ff{g.ia0h, g.ia0l}), ff{g.ib0h, g.ib0l});
    int f = at.y;
    unsigned p = 3;
    for (int iv = 0; iv < M - 3; iv++) {
        if (at.x + p >= nword) {                            // (the guard words are more than any cloud takes)
            atomicOr(err, WS_LOST);
            return;
        }
        int hv;
        ff n;
        double slow = 0.0;
        const bool one = ws_fast(w[p], kn, hv);
        if (one) {
            const float2 t = wnf[hv & 127];
            const int h16 = hv >> 16;                       // hv = 65536 h16 + l16, both exact in float32
            const float fh = __fsub_rn(__int_as_float(0x4B400000 + h16), BB_MAGIC15) * 65536.0f;
            const float fl = __fsub_rn(__int_as_float(0x4B400000 + (hv & 0xffff)), BB_MAGIC15);
            n = ff_mul(ff_two_sum(fh, fl), ff{t.x, t.y});
            p++;
        } else {
            while (f < cap - 1 && fpos[f] < at.x + p) f++;  // (words inside an earlier deviate, or uniform draws)
            slow = fval[f];
            n = ff_of(slow);
            p += 1 + fext[f];
            f++;
        }
        int c;
        if (!g.fast_ok || !ff_round(ff_add(ch0, ff_mul(n, chw)), c)) c = -0x40000000;
        for (int nl = 0; nl < g.nlines; nl++) {
            long long kc = c;
            if (nl || c == -0x40000000) {
                const double d = one ? __dmul_rn((double)hv, zig->wn[hv & 127]) : slow;
                const double v = __dadd_rn(vs, __dmul_rn(d, s.vdisp)), ch = velgrid_exact(v, g, nl);
                kc = lround_ref(ch);
                if (ws_close(ch)) {
                    // (the velocity is within dv of the one from the C library's functions)
                    const double dv = 1e-14 * (fabs(s.vsys) + 4.0 * (fabs(s.vsph) + fabs(s.vrot)) + 16.0 * fabs(s.vdisp));
                    if (lround_ref(velgrid_exact(__dsub_rn(v, dv), g, nl)) != kc ||
                        lround_ref(velgrid_exact(__dadd_rn(v, dv), g, nl)) != kc)
                        atomicOr(err, WS_NEAR);
                }
            }
            if (kc < 0 || kc >= g.nz) continue;
            atomicAdd(o + kc, (unsigned long long)fx[(size_t)nl * g.nz + kc]);
        }
    }
}

// the sums (by, bx, nz) as the cube (nz, by, bx) in float64
__global__ void k_ws_cube(const long long *__restrict__ acc, long long npix, int nz, double unit,
                          double *__restrict__ out) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    for (int k = 0; k < nz; k++) out[(size_t)k * npix + p] = __dmul_rn((double)acc[p * nz + k], unit);
}

}  // namespace

void launch_wind_mc(cudaStream_t st, const WindShell *shells, const int *shell, const double *geo,
                    const long long *nbase, const long long *sbase, const int *hz, const double *slow,
                    const ZigDev *zig, long long ncloud, const GridDev &g, const double *cd2i, int blo0, int blo1,
                    int bhi0, int bhi1, double scale, unsigned long long *acc) {
    if (ncloud <= 0) return;
    k_wind_mc<<<(unsigned)((ncloud + 255) / 256), 256, 0, st>>>(shells, shell, geo, nbase, sbase, hz, slow, zig, ncloud,
                                                                 g, cd2i, blo0, blo1, bhi0, bhi1, scale, acc);
}

void launch_ws_words(cudaStream_t st, const WindJob *jobs, int njob, int nseg, const void *jump, const ZigDev *zig,
                     const double *fn, unsigned long long *words, unsigned *masks, int *nfail, int *foff, int *fcur,
                     int *scratch, unsigned *fpos, unsigned char *fext, double *fval, int cap, int *err) {
    k_ws_gen<<<(nseg + 127) / 128, 128, 0, st>>>(jobs, njob, nseg, (const ulonglong2 *)jump, zig, words, masks, nfail);
    launch_scan_tiles(st, nfail, foff, fcur, nseg, scratch);
    const int nmask = nseg * (WS_SEG / 32);
    k_ws_list<<<(nmask + 255) / 256, 256, 0, st>>>(masks, nmask, foff, fpos, cap, err);
    k_ws_slow<<<(cap + 127) / 128, 128, 0, st>>>(fpos, foff, nseg, nfail, cap, words, (unsigned)nseg * WS_SEG, zig, fn,
                                                 fext, fval, err);
}

void launch_ws_clouds(cudaStream_t st, const WindJob *jobs, int njob, int nblk, int ngrp, long long ncl, int M,
                      const int *foff, const unsigned *fpos, const unsigned char *fext, const double *fval, int cap,
                      unsigned *spec, WsStart *group, WsStart *start, WsStart *ends, void *cloud,
                      const unsigned long long *words, unsigned nword, const ZigDev *zig, const WindShell *shells,
                      const WindCloudLaw *law, const long long *sfirst, int *err, const GridDev &g, int blo0, int blo1,
                      int bhi0, int bhi1, const long long *fix, unsigned long long *acc) {
    WsStart *gstart = group + (size_t)ngrp * M;
    k_ws_spec<<<(unsigned)(((long long)nblk * M + 255) / 256), 256, 0, st>>>(jobs, njob, nblk, M, foff, fpos, fext, cap,
                                                                             spec);
    k_ws_group<<<(unsigned)(((long long)ngrp * M + 63) / 64), 64, 0, st>>>(jobs, njob, ngrp, M, foff, fpos, fext, cap,
                                                                           spec, group);
    k_ws_chain<<<njob, 32, 0, st>>>(jobs, njob, M, foff, fpos, fext, cap, spec, group, gstart, ends);
    k_ws_expand<<<(ngrp + 31) / 32, 32, 0, st>>>(jobs, njob, ngrp, M, foff, fpos, fext, cap, spec, gstart, start);
    k_ws_place<<<(nblk + 63) / 64, 64, 0, st>>>(jobs, njob, nblk, M, foff, fpos, fext, cap, start, (uint2 *)cloud);
    k_ws_clouds<<<(unsigned)((ncl + 255) / 256), 256, 0, st>>>(jobs, njob, ncl, M, ends, (const uint2 *)cloud, words,
                                                               fpos, fext, fval, zig, shells, law, sfirst, nword, cap,
                                                               err, g, blo0, blo1, bhi0, bhi1, fix, acc);
}

void launch_ws_flux(cudaStream_t st, const WindShell *shells, int nshell, const GridDev &g, const double *cd2i,
                    double scale, long long *fix) {
    const long long n = (long long)nshell * g.nlines * g.nz;
    if (n) k_ws_flux<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(shells, nshell, g, cd2i, scale, fix);
}

void launch_ws_cube(cudaStream_t st, const unsigned long long *acc, long long npix, int nz, double unit, double *out) {
    if (npix) k_ws_cube<<<(unsigned)((npix + 127) / 128), 128, 0, st>>>((const long long *)acc, npix, nz, unit, out);
}
