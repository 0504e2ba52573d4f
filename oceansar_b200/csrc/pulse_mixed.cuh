// Mixed-precision pulse kernel (sm_100a): the body of the azimuth loop of sar_raw
// (oceansar/radarsim/sar_raw_nompi.py:349-535) for SAR scenes with Kodis specular and / or
// Romeiser Bragg scattering, in the split-range precision form:
//
//   float64 only per pulse row and per column (the reference ranges):
//     R_y = az/2 * sin_az (row), sr_c = slant range of the column, both reduced to
//     2 k0 R mod 2 pi and converted to range-bin units, split into a float32 high part on a
//     2^-8-bin grid (so that high parts add exactly) and a float32 low part;
//   float32 per facet (the bulk):
//     delta = -cos_inc Dz + Dx sin_inc + Dy sin_az (the facet's range offset), the bin
//     position hi + (lo + delta / binsize) and the two-way phase
//     phi_col + phi_row - 2 k0 delta, whose large product 2 k0 delta is reduced exactly
//     (an error-free product and a three-part 2 pi), the Kodis field, the Bragg lines,
//     antenna / ATI / XTI factors and the accumulation;
//   float64 only for facets whose float32 decision is within its error bound of a
//     rounding boundary (range bin floor, LUT round-half-even, Kodis facet window), which
//     are re-decided with the float64 drop-in's exact arithmetic: bins, LUT indices and
//     specular facet selection are therefore identical to the float64 form's.
//
// Two forms of the accumulation, chosen by the geometry (mixed_hist_ok):
//
// * Fine grid (mix_hist_tile; scenes whose 128-column tiles span few range bins): a facet's
//   taps depend only on its (bin, LUT index) cell, so each facet adds its coefficient of
//   every output once into a shared-memory grid H[bin][LUT index] (float32 shared atomic
//   adds), and the tile's H is convolved with the pulse once, at its end, and added to the
//   complex64 raw row with compensated global atomics whose rounding errors collect in a
//   per-pulse float32 compensation row, which the launch's last CTA folds into the raw row.
// * Register windows (mix_tile; wide tiles): 12-slot windows per thread (float32 FMA; a
//   window sums at most one tile height of facets), flushed into CTA shared bins kept as
//   compensated (hi, lo) float32 pairs (TwoSum of every shared atomic add), added to the
//   raw row the same way; here the next pulse's row-table kernel (or ocs_pulse_flush) folds
//   the compensation row.
//
// Input staging of the register-window form: the facet inputs of a CTA row (the float32
// fields, sqrt(RCS) and scatterer start indices of 128 columns) are moved into a four-row
// shared-memory ring by tiled tensor copies (cp.async.bulk.tensor: one three-dimensional box
// for all fields, one per index map and one for the sqrt(RCS) planes) that complete on the
// slot's mbarrier.  The warp that finishes reading a row last refills its slot with the row
// four ahead, so no warp ever waits for another, only for data.  Every mbarrier wait is
// bounded: a wait that gives up sets the launch's error flag, lets the copies in flight land
// and ends the CTA's work.  The fine-grid form, which needs half the registers, reads its
// inputs straight into registers one row ahead.
#pragma once
#include <cuda.h>

#include "bulk.cuh"
#include "pulse_core.cuh"

namespace ocs {

constexpr int kMixCols = 128;       // columns (threads) per CTA, 32 per warp
constexpr int kMixSlots = 4;        // ring rows (three in flight while one is read)
constexpr int kMixArrays = 14;      // staged input arrays per row (see MixArr)
constexpr int kMixRT = 8;           // float row-table entries before the channel factors
constexpr int kHistThreads = 256;   // threads of a fine-grid CTA: 128 columns x 2 rows
constexpr int kHistStreams = kHistThreads / kMixCols;
constexpr int kMixS = 12;           // register-window slots
constexpr int kMixNbw = 160;        // CTA shared bin window

// staged arrays: fields, Kodis curvatures, scatterer start indices, sqrt(RCS) [pol][line]
enum MixArr { kAdx = 0, kAdy, kAdz, kAdiffx, kAdiffy, kAdxx, kAdyy, kAdxy, kAindm, kAindp, kAscat };

// Tensor maps of one launch's inputs: the fields as one [nf][ny][nx] float32 tensor (the
// surface keeps them in one block, Dx Dy Dz Diffx Diffy [Diffxx Diffyy Diffxy]), the two
// int32 [ny][nx] scatterer index maps and the [2 npol][ny][nx] sqrt(RCS) planes; every box
// is one row of kMixCols columns.
struct alignas(64) MixMaps {
    CUtensorMap fields, indm, indp, scat;
    int nf;                         // fields in the fields map (5, or 8 with the curvatures)
};

// Per-pulse workspace after the float64 row table: float row table [ny][mix_rt(nch)]
// (Bh, Bl, phi_y, sin_az, cos_azp, sin_azp, -, -, then the channel factors, padded to
// 16 bytes), then the header {pending raw row, error flag, CTAs done}.
OCS_HD int mix_rt(int nch) { return kMixRT + ((2 * nch + 3) & ~3); }
OCS_HD size_t mix_rowtab_offset(int ny, int nch) {
    return ((size_t)ny * (5 + 2 * nch) * sizeof(double) + 15) & ~(size_t)15;
}
OCS_HD size_t mix_hdr_offset(int ny, int nch) {
    return (mix_rowtab_offset(ny, nch) + (size_t)ny * mix_rt(nch) * sizeof(float) + 15) & ~(size_t)15;
}
constexpr size_t kMixHdrBytes = 16;
// Floats of a tile's row (MixRow): 6 terms and the factors, a multiple of 4.
template <int NOUT> OCS_HD constexpr int mix_row_floats() { return (6 + 2 * NOUT + 3) & ~3; }

// ---------------------------------------------------------------------------------------
// Split-float helpers.
OCS_D float two_sum_err(float a, float b, float s) {
    const float bp = __fsub_rn(s, a);
    return __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// Compensated add of v into the shared pair (hi, lo): the atomic returns the old high
// part, from which the exact rounding error of the stored sum follows.
OCS_D void cadd_shared(float *hi, float *lo, float v) {
    if (v == 0.f) return;
    const float old = atomicAdd(hi, v);
    const float err = two_sum_err(old, v, __fadd_rn(old, v));
    if (err != 0.f) atomicAdd(lo, err);
}

// Reduction of a float32 phase p = K_hi * d (plus the exact product error and K_lo * d) to
// about [-pi, pi]: n = rint(p / 2 pi), p - n P1 exactly (P1 has 8 significant bits), then
// the remaining parts of 2 pi.
OCS_D float reduce_prod(float khi, float klo, float d) {
    const float p = __fmul_rn(khi, d);
    const float pe = fmaf(khi, d, -p) + klo * d;
    const float n = rintf(p * 0.15915494309189535f);
    float r = fmaf(-n, 6.28125f, p);                      // exact
    r = fmaf(-n, 1.9353071693331003e-3f, r);              // 2 pi - 6.28125, float part
    r = fmaf(-n, 1.0253376273028358e-11f, r);             // remainder of 2 pi
    return r + pe;
}
OCS_D float wrap_pi(float x) { return fmaf(-rintf(x * 0.15915494309189535f), 6.2831853071795865f, x); }

// Split of a float64 bin position into a float32 part on a 2^-8 grid and a float32 rest.
OCS_HD void split_bins(double v, float &hi, float &lo) {
    const double h = rint(v * 256.0) * (1.0 / 256.0);
    hi = (float)h;
    lo = (float)(v - h);
}

// ---------------------------------------------------------------------------------------
// Per-pulse row tables of the mixed kernel: the float64 table of pulse_row plus the float
// table (split bin position and reduced phase of R_y, sin_az, projected azimuth cos / sin,
// channel factors).  Threads beyond the rows fold the previous pulse's compensation
// row into its raw row.
OCS_D void mix_row(const PulseArgs &a, double az_now, int y) {
    unsigned char *ws = reinterpret_cast<unsigned char *>(a.rowtab);
    pulse_row(a, az_now, y);
    {
        const double az = a.rowtab[y], sin_az = a.rowtab[(long long)a.ny + y];
        const double ry = dmul(az * 0.5, sin_az);
        float *ft = reinterpret_cast<float *>(ws + mix_rowtab_offset(a.ny, a.nch)) + (long long)y * mix_rt(a.nch);
        split_bins(ry * a.inv_binsize, ft[0], ft[1]);
        ft[2] = (float)reduce_2pi((-2.0 * a.k0) * ry);
        ft[3] = (float)sin_az;
        ft[4] = (float)a.rowtab[3LL * a.ny + y];
        ft[5] = (float)a.rowtab[4LL * a.ny + y];
        const double *fac = a.rowtab + 5LL * a.ny + 2LL * y * a.nch;
        for (int c = 0; c < 2 * a.nch; ++c) ft[kMixRT + c] = (float)fac[c];
    }
}

// ---------------------------------------------------------------------------------------
// Shared memory of the mixed kernel.
template <int NOUT> struct MixSmem {
    float *wtab;                    // pre-shifted weights [5][21][12]
    float *bhi, *blo;               // CTA bins [NOUT][kMixNbw][2] (hi, lo)
    float *rt;                      // rows of the tile [rows][mix_row_floats]
    double *raz;                    // their float64 azimuth terms [rows][4]
    double *sred;                   // block reduction scratch [32]
    float *stage;                   // [kMixSlots][kMixArrays][kMixCols]
    unsigned long long *bar;        // [kMixSlots] full barriers
    int *cnt;                       // [kMixSlots] warps done with the slot's row
};

template <int NOUT> OCS_HD size_t mix_smem_bytes(int nch, int rows_cap) {
    return (size_t)wtab_len<float, kMixS>(kSincTaps, kSincOvs) * 4 + (size_t)NOUT * kMixNbw * 2 * 2 * 4 +
           (size_t)rows_cap * (mix_row_floats<NOUT>() * 4 + 4 * 8) + 32 * 8 +
           (size_t)kMixSlots * kMixArrays * kMixCols * 4 + kMixSlots * 16 + 256;
}

template <int NOUT> OCS_D MixSmem<NOUT> mix_smem(unsigned char *smem, int nch, int rows_cap) {
    MixSmem<NOUT> sm;
    size_t off = 0;
    auto take = [&](size_t bytes, size_t align) {
        off = (off + align - 1) & ~(align - 1);
        unsigned char *p = smem + off;
        off += bytes;
        return p;
    };
    sm.bar = reinterpret_cast<unsigned long long *>(take(kMixSlots * 8, 8));
    sm.cnt = reinterpret_cast<int *>(take(kMixSlots * 4, 4));
    sm.stage = reinterpret_cast<float *>(take((size_t)kMixSlots * kMixArrays * kMixCols * 4, 128));
    sm.wtab = reinterpret_cast<float *>(take((size_t)wtab_len<float, kMixS>(kSincTaps, kSincOvs) * 4, 16));
    sm.bhi = reinterpret_cast<float *>(take((size_t)NOUT * kMixNbw * 2 * 4, 16));
    sm.blo = reinterpret_cast<float *>(take((size_t)NOUT * kMixNbw * 2 * 4, 16));
    sm.rt = reinterpret_cast<float *>(take((size_t)rows_cap * mix_row_floats<NOUT>() * 4, 16));
    sm.raz = reinterpret_cast<double *>(take((size_t)rows_cap * 4 * 8, 8));
    sm.sred = reinterpret_cast<double *>(take(32 * 8, 8));
    return sm;
}

// Register window of one thread (accum.cuh's BinWindow, flushed into compensated bins).
template <int NOUT> struct MixBins {
    float *hi, *lo;                 // shared [NOUT][kMixNbw][2]
    int cta_base, nout, nbins;
    float *out;                     // raw row of output 0 (complex64 interleaved)
    float *lo_row;                  // compensation row of output 0, or null
    long long out_stride;           // floats between outputs in out

    // bins outside the CTA window: compensated global atomics
    OCS_D void add_global(int o, int b, float re, float im) {
        float *d = out + (long long)o * out_stride + 2 * b;
        if (re != 0.f) {
            const float old = atomicAdd(d, re);
            const float e = two_sum_err(old, re, __fadd_rn(old, re));
            if (lo_row && e != 0.f) atomicAdd(lo_row + (long long)o * 2 * nbins + 2 * b, e);
        }
        if (im != 0.f) {
            const float old = atomicAdd(d + 1, im);
            const float e = two_sum_err(old, im, __fadd_rn(old, im));
            if (lo_row && e != 0.f) atomicAdd(lo_row + (long long)o * 2 * nbins + 2 * b + 1, e);
        }
    }
    OCS_D void add(int o, int b, float re, float im) {
        if (o >= nout || b < 0 || b >= nbins) return;
        const int lb = b - cta_base;
        if (lb >= 0 && lb < kMixNbw) {
            const int i = 2 * (o * kMixNbw + lb);
            cadd_shared(hi + i, lo + i, re);
            cadd_shared(hi + i + 1, lo + i + 1, im);
        } else {
            add_global(o, b, re, im);
        }
    }
};

template <int NOUT> struct MixWindow {
    float re[NOUT][kMixS], im[NOUT][kMixS];
    int base, lo, hi;
    bool live;

    OCS_D void reset() {
#pragma unroll
        for (int o = 0; o < NOUT; ++o)
#pragma unroll
            for (int s = 0; s < kMixS; ++s) { re[o][s] = 0.f; im[o][s] = 0.f; }
        live = false;
        lo = kMixS;
        hi = -1;
    }
    OCS_D void flush(MixBins<NOUT> &cb) {
        if (!live) return;
#pragma unroll
        for (int s = 0; s < kMixS; ++s) {
            if (s >= lo && s <= hi) {
#pragma unroll
                for (int o = 0; o < NOUT; ++o) cb.add(o, base + s, re[o][s], im[o][s]);
            }
        }
        reset();
    }
    // facet whose first tap is bin `first`, LUT index `lut`
    OCS_D void add(int first, int lut, const c64 (&coef)[NOUT], const float *wtab, const float *sinc,
                   MixBins<NOUT> &cb) {
        float sum = 0.f;
#pragma unroll
        for (int o = 0; o < NOUT; ++o) sum += coef[o].re + coef[o].im;
        if (!isfinite(sum)) {
            // non-finite coefficients touch exactly their own taps, as in the reference
            for (int j = 0; j < kSincTaps; ++j) {
                const float w = sinc[lut + j * kSincOvs];
#pragma unroll
                for (int o = 0; o < NOUT; ++o)
                    cb.add(o, first + j, w * coef[o].re - 0.f * coef[o].im, w * coef[o].im + 0.f * coef[o].re);
            }
            return;
        }
        constexpr int slack = kMixS - kSincTaps;
        int off = first - base;
        if (!live || off < 0 || off > slack) {
            flush(cb);
            base = first - slack / 2;
            off = slack / 2;
            live = true;
        }
        lo = min(lo, off);
        hi = max(hi, off + kSincTaps - 1);
        const float4 *w = reinterpret_cast<const float4 *>(wtab + (off * (kSincOvs + 1) + lut) * wtab_stride<float, kMixS>());
#pragma unroll
        for (int v = 0; v < kMixS / 4; ++v) {
            const float4 wv = w[v];
            const float ws[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int s = 4 * v + k;
#pragma unroll
                for (int o = 0; o < NOUT; ++o) {
                    re[o][s] = fmaf(ws[k], coef[o].re, re[o][s]);
                    im[o][s] = fmaf(ws[k], coef[o].im, im[o][s]);
                }
            }
        }
    }
};

// Tile-end flush of a warp's 32 register windows without contention: every lane writes its
// window (one output at a time) into the warp's scratch, then lane l sums bin lo + l (and
// every 32nd after it) over the lanes whose windows cover it, in lane order, and makes one
// compensated add into the CTA bins -- the lanes of a warp never add to the same bin.
// scr: per-warp [32][kMixS][2] floats; sbase: per-warp [32] ints.  All 32 lanes call it.
template <int NOUT>
OCS_D void warp_flush(MixWindow<NOUT> &win, MixBins<NOUT> &cb, float *scr, int *sbase) {
    const int lane = threadIdx.x & 31;
    int lo = win.live ? win.base + win.lo : 0x3fffffff;
    int hi = win.live ? win.base + win.hi : -0x3fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (hi < lo) return;                  // no live window in the warp
    sbase[lane] = win.live ? win.base : -0x3fffffff;
#pragma unroll
    for (int o = 0; o < NOUT; ++o) {
#pragma unroll
        for (int sl = 0; sl < kMixS; ++sl) {
            scr[(lane * kMixS + sl) * 2] = win.re[o][sl];
            scr[(lane * kMixS + sl) * 2 + 1] = win.im[o][sl];
        }
        __syncwarp();
        for (int b = lo + lane; b <= hi; b += 32) {
            float sr = 0.f, si = 0.f;
            for (int j = 0; j < 32; ++j) {
                const int off = b - sbase[j];
                if (off >= 0 && off < kMixS) {
                    sr += scr[(j * kMixS + off) * 2];
                    si += scr[(j * kMixS + off) * 2 + 1];
                }
            }
            cb.add(o, b, sr, si);
        }
        __syncwarp();
    }
    win.reset();
}

// Float64 slant range of one facet exactly as the drop-in computes it (no contraction).
OCS_D double srs_f64(double sr_c, double cos_i, double sin_i, double az, double sin_az, float dx, float dy,
                     float dz) {
    double srs = dsub(sr_c, dmul(cos_i, (double)dz));
    srs = dadd(srs, dmul(az * 0.5, sin_az));
    srs = dadd(srs, dmul((double)dx, sin_i));
    return dadd(srs, dmul((double)dy, sin_az));
}

// Constants of one column: float64 reference quantities, converted once.
struct MixCol {
    float Ch, Cl, phi_x, sin_i, cos_i, tan_i, dinc0, cap_r;

    template <bool KODIS, int FAST> OCS_D void init(const PulseArgs &a, int xs) {
        const double sr_c = a.sr_col[xs];
        split_bins((sr_c - a.min_sr) * a.inv_binsize, Ch, Cl);
        phi_x = (float)reduce_2pi((-2.0 * a.k0) * sr_c);
        sin_i = (float)a.sin_inc[xs];
        cos_i = (float)a.cos_inc[xs];
        tan_i = (FAST || (KODIS && a.do_kodis)) ? (float)a.tan_inc[xs] : 0.f;
        dinc0 = (float)(a.inc[xs] - a.inc_angle);
        cap_r = 0.f;
        if (a.do_bragg) cap_r = (float)reduce_2pi(((2.0 * a.k0) * a.t_step) * a.c_b[xs] * (double)(a.az_step + 1));
    }
};

// One row of the pass: position, phase and azimuth terms, the outputs' factors, and the float64
// azimuth terms of the re-decisions {az, sin_az, cos_azp, sin_azp}.
template <int NOUT> struct MixRow {
    float Bh, Bl, phi, sin_az, cos_azp, sin_azp;
    float fac[2 * NOUT];
    const double *exact;
    OCS_D void load(const float *row, const double *ex) {
        const float4 p = *reinterpret_cast<const float4 *>(row), q = *reinterpret_cast<const float4 *>(row + 4);
        Bh = p.x; Bl = p.y; phi = p.z; sin_az = p.w;
        cos_azp = q.x; sin_azp = q.y;
        fac[0] = q.z; fac[1] = q.w;
#pragma unroll
        for (int k = 2; k < 2 * NOUT; k += 2) {
            const float2 v = *reinterpret_cast<const float2 *>(row + 6 + k);
            fac[k] = v.x; fac[k + 1] = v.y;
        }
        exact = ex;
    }
    // float part of a row from its float64 quantities (the first factor sits in entries 6, 7)
    static OCS_D void store(float *row, const PulseArgs &a, double az, double sin_az, double cos_azp, double sin_azp) {
        const double ry = dmul(az * 0.5, sin_az);
        split_bins(ry * a.inv_binsize, row[0], row[1]);
        row[2] = (float)reduce_2pi((-2.0 * a.k0) * ry);
        row[3] = (float)sin_az;
        row[4] = (float)cos_azp;
        row[5] = (float)sin_azp;
    }
};

// Outputs of a pass, 5 bits each: channel, polarisation, XTI flag.
template <int NOUT> OCS_D unsigned mix_outs(const PulseArgs &a) {
    unsigned outs = 0;
#pragma unroll
    for (int k = 0; k < NOUT; ++k) {
        const int o = a.out0 + k;
        const int p = o / a.nch, c = o - p * a.nch;
        const bool xti = k < a.nout && a.b_xti[c] != 0.0;
        outs |= (unsigned)(c | (p << 3) | (xti ? 16 : 0)) << (5 * k);
    }
    return outs;
}

// Inputs of one facet: fields, sqrt(RCS) of both Bragg lines per polarisation, and the
// scatterer-series values of the two lines.
struct MixIn {
    float dx = 0.f, dy = 0.f, dz = 0.f, diffx = 0.f, diffy = 0.f, dxx = 0.f, dyy = 0.f, dxy = 0.f;
    float sc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    float2 cm = {0.f, 0.f}, cp = {0.f, 0.f};
};

// Range bin, LUT index and coefficient of every output of a facet in column x; outs: mix_outs.
template <int NOUT, bool KODIS, int FAST>
OCS_D void mix_facet(const PulseArgs &a, const MixCol &c, const MixIn &in, const MixRow<NOUT> &row,
                     unsigned outs, int x, int &bin_d, int &lut, c64 (&coef)[NOUT], double &spec_sum) {
    const bool kodis = FAST || (KODIS && a.do_kodis);
    const bool bragg = FAST || a.do_bragg;
    const int npol = FAST ? 1 : a.npol;
    const float sin_az = row.sin_az;
    // ---- range offset, bin and LUT index ----
    const float delta = fmaf(in.dy, sin_az, fmaf(in.dx, c.sin_i, -(c.cos_i * in.dz)));
    const float S = c.Ch + row.Bh;                                   // exact
    const float r = fmaf(delta, a.f_inv_bs, c.Cl + row.Bl);
    float fl = floorf(S + r);
    float frac = (S - fl) + r;
    if (frac < 0.f) { fl -= 1.f; frac += 1.f; }
    else if (frac >= 1.f) { fl += 1.f; frac -= 1.f; }
    const float x20 = fmaf(-20.f, frac, 20.f);
    float lutf = rintf(x20);
    // error bound of frac (float32 delta and rounding), with a wide margin
    const float eb = 4.76837158e-7f * ((fabsf(in.dz) + fabsf(in.dx) + fabsf(in.dy)) * a.f_inv_bs + fabsf(r) + 2.f);
    const bool finite = fabsf(fl) < 1.0e9f;
    if (!finite || frac < eb || frac > 1.f - eb || fabsf(fabsf(x20 - lutf) - 0.5f) < 20.f * eb + 1e-6f) {
        // near a rounding boundary (or not finite): the float64 drop-in's decision
        const double srs = srs_f64(a.sr_col[x], a.cos_inc[x], a.sin_inc[x], row.exact[0], row.exact[1],
                                   in.dx, in.dy, in.dz);
        bin_and_lut(srs, a.min_sr, a.binsize, kSincOvs, bin_d, lut);
    } else {
        bin_d = (int)fl;
        lut = (int)lutf;
    }
    // ---- two-way phase of the facet: phi_x + phi_y - 2 k0 delta ----
    const float th = wrap_pi((c.phi_x + row.phi) - reduce_prod(a.f_khi, a.f_klo, delta));

    c64 scene[2] = {{0.f, 0.f}, {0.f, 0.f}};
    if (kodis) {
        // Kodis stationary point of the facet (kodis.py:38-73) in float32
        const float J = __fsub_rn(__fmul_rn(in.dxx, in.dyy), __fmul_rn(in.dxy, in.dxy));
        if (J != 0.f) {
            const float Ja = fabsf(J);
            const float inv_j = __fdividef(1.f, Ja);
            const float cos_azp = row.cos_azp, sin_azp = row.sin_azp;
            const float ty = in.diffy - c.tan_i * sin_azp;
            const float tx = in.diffx - c.tan_i * cos_azp;
            const float ddx = inv_j * (in.dxy * ty - in.dyy * tx);
            const float ddy = inv_j * (in.dxy * tx - in.dxx * ty);
            const float keb = 7.62939453e-6f * inv_j * (fabsf(in.dxx) + fabsf(in.dyy) + 2.f * fabsf(in.dxy)) *
                              (fabsf(tx) + fabsf(ty) + fabsf(in.diffx) + fabsf(in.diffy) + c.tan_i) + 1e-30f;
            bool inside = (fabsf(ddx) < a.f_hdx) && (fabsf(ddy) < a.f_hdy);
            if (fabsf(fabsf(ddx) - a.f_hdx) < keb || fabsf(fabsf(ddy) - a.f_hdy) < keb) {
                // near the facet window: the float64 drop-in's test
                const double ij = (double)(1.f / Ja);
                const double tan_d = a.tan_inc[x];
                const double tyd = (double)in.diffy - tan_d * row.exact[3];
                const double txd = (double)in.diffx - tan_d * row.exact[2];
                const double dxd = ij * ((double)in.dxy * tyd - (double)in.dyy * txd);
                const double dyd = ij * ((double)in.dxy * txd - (double)in.dxx * tyd);
                inside = (-a.kodis.hdx < dxd) && (dxd < a.kodis.hdx) && (-a.kodis.hdy < dyd) &&
                         (dyd < a.kodis.hdy);
            }
            if (inside) {
                const float ddz = ddx * in.diffx + ddy * in.diffy;
                const float off = c.sin_i * cos_azp * ddx + c.sin_i * sin_azp * ddy - c.cos_i * ddz;
                const float ph = wrap_pi((c.phi_x + row.phi) - reduce_prod(a.f_khi, a.f_klo, delta + off));
                float s, co;
                __sincosf(ph, &s, &co);
                const float sgn = J > 0.f ? (float)((in.dxx > 0.f) - (in.dxx < 0.f)) : 0.f;
                const float fac =
                    __fadd_rn(__fadd_rn(__fmul_rn(in.diffx, in.diffx), __fmul_rn(in.diffy, in.diffy)), 1.f);
                const float amp = fac * 3.5449077018110318f / sqrtf(Ja);    // sqrt(4 pi)
                // (R/2) eps fac e^{i ph} / sqrt|J|, eps = sign(Dxx) or 1j
                const c64 re = J > 0.f ? c64{a.f_hr * sgn, a.f_hi * sgn} : c64{-a.f_hi, a.f_hr};
                const c64 e = cmul(re, c64{co * amp, s * amp});
                spec_sum += (double)e.re * e.re + (double)e.im * e.im;
                scene[0] = e;
                scene[1] = e;
            }
        }
    }
    if (bragg) {
        // Bragg phases -2 k0 r -/+ 2 k0 t_step c_b (az_step + 1)
        float s0, c0, s1, c1;
        __sincosf(th - c.cap_r, &s0, &c0);
        __sincosf(th + c.cap_r, &s1, &c1);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            if (p < npol) {
                const c64 l0 = cmul(c64{in.sc[p][0] * c0, in.sc[p][0] * s0}, c64{in.cm.x, in.cm.y});
                const c64 l1 = cmul(c64{in.sc[p][1] * c1, in.sc[p][1] * s1}, c64{in.cp.x, in.cp.y});
                scene[p] = cadd(scene[p], cadd(l0, l1));
            }
        }
    }
    // ---- channels: antenna pattern x ATI phase (row) x XTI phase (facet) ----
    float wave_dinc = 0.f;
    if (FAST == 2 || (FAST == 0 && a.any_xti)) wave_dinc = (in.dz * c.sin_i + in.dx * c.sin_i) * a.f_inv_sr0;
#pragma unroll
    for (int k = 0; k < NOUT; ++k) {
        if (FAST || k < a.nout) {
            // fast configurations: one polarisation, output k is channel out0 + k (mode 1:
            // no XTI phase; mode 2: the XTI flags of the tile's output word)
            const unsigned okb = FAST == 1 ? (unsigned)(a.out0 + k) : outs >> (5 * k);
            const int ch = okb & 7;
            const c64 f = {row.fac[2 * k], row.fac[2 * k + 1]};
            c64 v = cmul((!FAST && (okb & 8)) ? scene[1] : scene[0], f);
            if (FAST != 1 && (okb & 16)) {
                const float ph = wrap_pi(a.f_kxti[ch] * (c.dinc0 + wave_dinc));
                float s, co;
                __sincosf(ph, &s, &co);
                v = cmul(v, c64{co, s});
            }
            coef[k] = v;
        } else {
            coef[k] = {0.f, 0.f};
        }
    }
}

// ---------------------------------------------------------------------------------------
// One tile of 128 columns x tile_rows rows.  `rseq` is the warp's running row count (ring
// slot and barrier parity); `bad` becomes true when a bounded wait gave up.
// TMA = false (the scene batch, whose slots keep no tensor maps): every thread stages its
// own column's inputs of each row into the same ring by per-thread asynchronous copies
// (cp.async, one group per row, four rows ahead) and waits only for its own copies, since
// it alone reads that column of a slot.
template <int NOUT, bool KODIS, bool TMA = true, int FAST = 0>
OCS_D void mix_tile(const PulseArgs &a, const MixMaps *maps, float *lo_row, int tile, int tile_rows,
                    const MixSmem<NOUT> &sm, unsigned &rseq, bool &bad, double &spec_sum) {
    const int lane = threadIdx.x & 31;
    const int tiles_x = (a.nx + kMixCols - 1) / kMixCols;
    const int x0t = (tile % tiles_x) * kMixCols;
    const int x = x0t + threadIdx.x;
    const int y0 = (tile / tiles_x) * tile_rows;
    const int nrows = min(tile_rows, a.ny - y0);
    constexpr int RT = mix_row_floats<NOUT>();
    __syncthreads();                      // the previous tile's bins and row tables are consumed
    for (int i = threadIdx.x; i < nrows; i += blockDim.x) {
        // rows of the per-pulse float and float64 tables, factors of the pass's outputs
        const float *ft = reinterpret_cast<const float *>(reinterpret_cast<const unsigned char *>(a.rowtab) +
                                                          mix_rowtab_offset(a.ny, a.nch)) +
                          (long long)(y0 + i) * mix_rt(a.nch);
        float *row = sm.rt + i * RT;
        for (int q = 0; q < 6; ++q) row[q] = ft[q];
        for (int k = 0; k < NOUT; ++k) {
            const int c = (a.out0 + min(k, a.nout - 1)) % a.nch;
            row[6 + 2 * k] = ft[kMixRT + 2 * c];
            row[7 + 2 * k] = ft[kMixRT + 2 * c + 1];
        }
        for (int q = 0; q < 4; ++q) sm.raz[4 * i + q] = a.rowtab[(long long)(q < 2 ? q : q + 1) * a.ny + y0 + i];
    }
    MixBins<NOUT> cb;
    cb.hi = sm.bhi;
    cb.lo = sm.blo;
    cb.nout = a.nout;
    cb.nbins = a.nbins;
    cb.out = reinterpret_cast<float *>(a.raw) + 2 * ((long long)a.out0 * a.raw_out_stride + a.raw_row);
    cb.lo_row = lo_row ? lo_row + 2LL * a.out0 * a.nbins : nullptr;
    cb.out_stride = 2 * a.raw_out_stride;
    {
        const int xc = min(x0t, a.nx - 1);
        const double az = (double)a.y[y0] - a.az_now;
        const double srg = a.sr_col[xc] + az * 0.5 * (az / a.sr0);
        cb.cta_base = (int)floor((srg - a.min_sr) / a.binsize) - 24;
    }
    for (int i = threadIdx.x; i < NOUT * kMixNbw * 2; i += blockDim.x) {
        sm.bhi[i] = 0.f;
        sm.blo[i] = 0.f;
    }
    __syncthreads();

    MixWindow<NOUT> win;
    win.reset();
    if (!bad) {
        // every warp takes part in every row (the ring's slots are released per warp);
        // lanes past the last column stage and wait but compute nothing
        const bool col_ok = x < a.nx;
        const int xs = col_ok ? x : a.nx - 1;
        MixCol col;
        col.init<KODIS, FAST>(a, xs);
        const unsigned outs = mix_outs<NOUT>(a);
        const bool kodis = FAST || (KODIS && a.do_kodis);
        const bool bragg = FAST || a.do_bragg;
        const int npol = FAST ? 1 : a.npol;
        const long long npix = (long long)a.nx * a.ny;
        float *scat = reinterpret_cast<float *>(a.scat);
        // ---- staging: tensor copies of whole CTA rows into the ring ----
        const int nf = TMA ? maps->nf : 0;
        const unsigned row_bytes = (unsigned)(nf + (a.do_bragg ? 2 + 2 * a.npol : 0)) * kMixCols * 4u;
        const unsigned first = rseq;      // ring position of this tile's row 0
        auto slot_of = [&](int r) { return (int)((first + (unsigned)r) % kMixSlots); };
        auto issue = [&](int r) {         // TMA: one thread; the slot of row r is free
            if constexpr (!TMA) {
                // every thread: its column's words of row r, one copy group per row (empty
                // past the tile, so that every thread counts the same groups)
                if (r < nrows) {
                    float *dst = sm.stage + (size_t)slot_of(r) * kMixArrays * kMixCols + threadIdx.x;
                    const long long g = (long long)(y0 + r) * a.nx + xs;
                    cp_async(dst + kAdx * kMixCols, a.dx_f + g, 4);
                    cp_async(dst + kAdy * kMixCols, a.dy_f + g, 4);
                    cp_async(dst + kAdz * kMixCols, a.dz_f + g, 4);
                    cp_async(dst + kAdiffx * kMixCols, a.diffx + g, 4);
                    cp_async(dst + kAdiffy * kMixCols, a.diffy + g, 4);
                    if (kodis) {
                        cp_async(dst + kAdxx * kMixCols, a.diffxx + g, 4);
                        cp_async(dst + kAdyy * kMixCols, a.diffyy + g, 4);
                        cp_async(dst + kAdxy * kMixCols, a.diffxy + g, 4);
                    }
                    if (bragg) {
                        cp_async(dst + kAindm * kMixCols, a.ind0_m + g, 4);
                        cp_async(dst + kAindp * kMixCols, a.ind0_p + g, 4);
                        cp_async(dst + kAscat * kMixCols, scat + g, 4);
                        cp_async(dst + (kAscat + 1) * kMixCols, scat + npix + g, 4);
                        if (npol == 2) {
                            cp_async(dst + (kAscat + 2) * kMixCols, scat + 2 * npix + g, 4);
                            cp_async(dst + (kAscat + 3) * kMixCols, scat + 3 * npix + g, 4);
                        }
                    }
                }
                cp_async_commit();
                return;
            }
            const int slot = slot_of(r);
            float *dst = sm.stage + (size_t)slot * kMixArrays * kMixCols;
            unsigned long long *bar = sm.bar + slot;
            fence_proxy_async();
            mbar_expect_tx(bar, row_bytes);
            const int yy = y0 + r;
            tma_load_3d(dst + kAdx * kMixCols, &maps->fields, x0t, yy, 0, bar);
            if (bragg) {
                tma_load_2d(dst + kAindm * kMixCols, &maps->indm, x0t, yy, bar);
                tma_load_2d(dst + kAindp * kMixCols, &maps->indp, x0t, yy, bar);
                tma_load_3d(dst + kAscat * kMixCols, &maps->scat, x0t, yy, 0, bar);
            }
        };
        auto wait_row = [&](int r) -> bool {
            if constexpr (!TMA) {
                // rows up to r + 3 are issued: row 0 waits with 3 groups pending, row r > 0
                // (waited at the top of row r - 1, with rows r + 1 and r + 2 issued) with 2
                if (r == 0) cp_async_wait<3>();
                else cp_async_wait<2>();
                return true;
            }
            const unsigned q = first + (unsigned)r;
            return mbar_wait(sm.bar + (q % kMixSlots), (q / kMixSlots) & 1u);
        };
        if (TMA && threadIdx.x == 0)
            for (int r = 0; r < kMixSlots && r < nrows; ++r) issue(r);
        if (!TMA)
            for (int r = 0; r < kMixSlots; ++r) issue(r);
        // gathers of the scatterer series, one row ahead
        float2 gm = {0.f, 0.f}, gp = {0.f, 0.f};
        const float2 *sm32 = reinterpret_cast<const float2 *>(a.s_m32);
        const float2 *sp32 = reinterpret_cast<const float2 *>(a.s_p32);
        auto gather = [&](int r, float2 &m, float2 &p) {
            const float *src = sm.stage + (size_t)slot_of(r) * kMixArrays * kMixCols;
            int i0 = __float_as_int(src[kAindm * kMixCols + threadIdx.x]);
            int i1 = __float_as_int(src[kAindp * kMixCols + threadIdx.x]);
            i0 += a.tmod_m;
            i0 = i0 >= a.n_m ? i0 - a.n_m : i0;
            i1 += a.tmod_p;
            i1 = i1 >= a.n_p ? i1 - a.n_p : i1;
            if (col_ok) {
                m = __ldg(sm32 + i0);
                p = __ldg(sp32 + i1);
            }
        };
        // every lane waits (acquiring the copied data), the warp agrees on the outcome
        int fail_row = -1;
        bool ok = __all_sync(0xffffffffu, wait_row(0));
        if (!ok) fail_row = 0;
        if (ok && bragg) gather(0, gm, gp);
        for (int i = 0; i < nrows && ok; ++i) {
            // rows i and i + 1 have landed
            if (i + 1 < nrows) {
                ok = __all_sync(0xffffffffu, wait_row(i + 1));
                if (!ok) { fail_row = i + 1; break; }
            }
            const int slot = slot_of(i);
            MixIn in;
            {
                const float *src = sm.stage + (size_t)slot * kMixArrays * kMixCols;
                const int t = threadIdx.x;
                in.dx = src[kAdx * kMixCols + t]; in.dy = src[kAdy * kMixCols + t]; in.dz = src[kAdz * kMixCols + t];
                in.diffx = src[kAdiffx * kMixCols + t]; in.diffy = src[kAdiffy * kMixCols + t];
                if (kodis) {
                    in.dxx = src[kAdxx * kMixCols + t];
                    in.dyy = src[kAdyy * kMixCols + t];
                    in.dxy = src[kAdxy * kMixCols + t];
                }
                if (bragg) {
                    in.sc[0][0] = src[kAscat * kMixCols + t];
                    in.sc[0][1] = src[(kAscat + 1) * kMixCols + t];
                    if (npol == 2) {
                        in.sc[1][0] = src[(kAscat + 2) * kMixCols + t];
                        in.sc[1][1] = src[(kAscat + 3) * kMixCols + t];
                    }
                }
            }
            in.cm = gm;
            in.cp = gp;
            if (bragg && i + 1 < nrows) gather(i + 1, gm, gp);
            // release the slot of row i; the last of the four warps refills it with row i + 4
            __syncwarp();
            if (TMA && lane == 0) {
                __threadfence_block();
                if (atomicAdd(sm.cnt + slot, 1) == 3) {
                    sm.cnt[slot] = 0;
                    __threadfence_block();
                    if (i + kMixSlots < nrows) issue(i + kMixSlots);
                }
            }
            if constexpr (!TMA) issue(i + kMixSlots);  // this thread's column of the slot is read
            if (!col_ok) continue;

            int bin_d, lut;
            c64 coef[NOUT];
            MixRow<NOUT> row;
            row.load(sm.rt + i * RT, sm.raz + 4 * i);
            mix_facet<NOUT, KODIS, FAST>(a, col, in, row, outs, x, bin_d, lut, coef, spec_sum);
            if (bin_d > -(1 << 29)) win.add(bin_d - kSincTaps / 2, lut, coef, sm.wtab, a.sinc, cb);
        }
        if (!ok) {
            // a wait gave up: record it, and let every copy that may be in flight (rows
            // fail_row .. fail_row + 3, one per slot) land before the shared memory can go away
            bad = true;
            if (lane == 0) {
                atomicOr(reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(a.rowtab) +
                                                 mix_hdr_offset(a.ny, a.nch)) + 1, 1);
                for (int r = fail_row; r < fail_row + kMixSlots && r < nrows; ++r) wait_row(r);
            }
            __syncwarp();
        }
        if constexpr (!TMA) cp_async_wait<0>();  // no copy may land in the ring after the tile
        rseq = first + (unsigned)nrows;
    }
    // every warp is past its last row: the ring holds no live data, its memory is the
    // flush scratch
    __syncthreads();
    {
        float *scr = sm.stage + (size_t)(threadIdx.x >> 5) * 32 * kMixS * 2;
        int *sbase = reinterpret_cast<int *>(sm.stage + (size_t)4 * 32 * kMixS * 2) + 32 * (threadIdx.x >> 5);
        warp_flush<NOUT>(win, cb, scr, sbase);
    }
    __syncthreads();
    // CTA bins -> raw row, compensated: first every returning add of this thread's bins (so
    // that their round trips overlap), then the rounding errors, as plain reductions, into
    // the compensation row
    constexpr int kPer = (NOUT * kMixNbw + kMixCols - 1) / kMixCols;
    float vr[kPer][2], orv[kPer][2], er[kPer][2];
    long long off[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int i = threadIdx.x + k * kMixCols;
        off[k] = -1;
        vr[k][0] = vr[k][1] = orv[k][0] = orv[k][1] = er[k][0] = er[k][1] = 0.f;
        if (i < a.nout * kMixNbw) {
            const int o = i / kMixNbw, lb = i - o * kMixNbw;
            const int b = cb.cta_base + lb;
            if (b >= 0 && b < a.nbins) {
                off[k] = (long long)o * cb.out_stride + 2 * b;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const float h = sm.bhi[2 * i + c], l = sm.blo[2 * i + c];
                    vr[k][c] = __fadd_rn(h, l);
                    er[k][c] = two_sum_err(h, l, vr[k][c]);
                    if (vr[k][c] != 0.f) orv[k][c] = atomicAdd(cb.out + off[k] + c, vr[k][c]);
                }
            }
        }
    }
    if (cb.lo_row) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (off[k] < 0) continue;
            const int i = threadIdx.x + k * kMixCols;
            const int o = i / kMixNbw, b = cb.cta_base + (i - o * kMixNbw);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (vr[k][c] == 0.f) continue;
                const float e = two_sum_err(orv[k][c], vr[k][c], __fadd_rn(orv[k][c], vr[k][c])) + er[k][c];
                if (e != 0.f) atomicAdd(cb.lo_row + (long long)o * 2 * a.nbins + 2 * b + c, e);
            }
        }
    }
}

template <int NOUT> OCS_D void mix_init(const MixSmem<NOUT> &sm) {
    if (threadIdx.x < kMixSlots) {
        mbar_init(sm.bar + threadIdx.x, 1);
        sm.cnt[threadIdx.x] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    __syncthreads();
}

// Record that the launch's compensation row belongs to this pulse's raw row.
OCS_D void mix_pending(const PulseArgs &a, float *lo_row) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && lo_row)
        reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(a.rowtab) + mix_hdr_offset(a.ny, a.nch))[0] =
            a.az_step;
}

template <int NOUT, bool KODIS, int FAST>
__global__ void __launch_bounds__(kMixCols, NOUT < 4 ? 4 : 2)
pulse_mixed_kernel(const __grid_constant__ PulseArgs a, const __grid_constant__ MixMaps maps, float *lo_row) {
    extern __shared__ __align__(128) unsigned char mix_raw[];
    const MixSmem<NOUT> sm = mix_smem<NOUT>(mix_raw, a.nch, kPulseRows);
    build_wtab<float, kMixS>(sm.wtab, a.sinc, kSincTaps, kSincOvs);
    mix_init<NOUT>(sm);
    const int tiles = ((a.nx + kMixCols - 1) / kMixCols) * ((a.ny + a.tile_rows - 1) / a.tile_rows);
    double spec_sum = 0.0;
    unsigned rseq = 0;
    bool bad = false;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
        mix_tile<NOUT, KODIS, true, FAST>(a, &maps, lo_row, tile, a.tile_rows, sm, rseq, bad, spec_sum);
    if (a.out0 == 0 && KODIS) block_atomic_sum(spec_sum, &a.nrcs_spec[a.az_step], sm.sred);
    mix_pending(a, lo_row);
}

// ---------------------------------------------------------------------------------------
// Fine-grid form.  Shared memory: the pulse's sinc table, H and the tile's row table.
template <int NOUT> struct HistSmem {
    double *sred;                   // block reduction scratch [32]
    double *tmp;                    // eval_tile_rows scratch [rows][2 + 2 NOUT]
    double *exact;                  // float64 azimuth terms of the tile's rows [rows][4]
    float *sinc;                    // [taps][kGridL]
    float *h;                       // [NOUT][re, im][kGridBins][kGridL]
    int *range;                     // touched rows of H of each warp [2][warps]
    float *rt;                      // rows of the tile [rows][mix_row_floats]
};

template <int NOUT> OCS_HD constexpr size_t hist_smem_bytes(int rows_cap) {
    return (32 + (size_t)rows_cap * (6 + 2 * NOUT)) * 8 +
           ((size_t)kSincTaps * kGridL + (size_t)NOUT * 2 * kGridBins * kGridL + 16 +
            (size_t)rows_cap * mix_row_floats<NOUT>()) * 4;
}

// Every part is a multiple of 16 bytes (rows_cap even).
template <int NOUT> OCS_D HistSmem<NOUT> hist_smem(unsigned char *smem, int rows_cap) {
    HistSmem<NOUT> sm;
    sm.sred = reinterpret_cast<double *>(smem);
    sm.tmp = sm.sred + 32;
    sm.exact = sm.tmp + rows_cap * (2 + 2 * NOUT);
    sm.sinc = reinterpret_cast<float *>(sm.exact + rows_cap * 4);
    sm.h = sm.sinc + kSincTaps * kGridL;
    sm.range = reinterpret_cast<int *>(sm.h + NOUT * 2 * kGridBins * kGridL);
    sm.rt = reinterpret_cast<float *>(sm.range + 16);
    return sm;
}

// H[bin][LUT index] of every output as separate real and imaginary planes, so that the lanes
// of one atomic add spread over all banks.  Facets outside H and non-finite coefficients
// (which must touch exactly their own taps) take per-tap global adds.
template <int NOUT, int FAST> struct MixHist {
    float *h;
    int base;                       // range bin of H's first row
    int tlo, thi;                   // rows of H this thread touched

    OCS_D void add(int bin_d, int lut, const c64 (&coef)[NOUT], const float *sinc, MixBins<NOUT> &cb) {
        float sum = 0.f;
#pragma unroll
        for (int o = 0; o < NOUT; ++o) sum += coef[o].re + coef[o].im;
        const int r = bin_d - base;
        if ((unsigned)r < (unsigned)kGridBins && isfinite(sum)) {
            float *c = h + r * kGridL + lut;
#pragma unroll
            for (int o = 0; o < NOUT; ++o) {
                if (FAST || o < cb.nout) {
                    atomicAdd(c + (2 * o) * kGridBins * kGridL, coef[o].re);
                    atomicAdd(c + (2 * o + 1) * kGridBins * kGridL, coef[o].im);
                }
            }
            tlo = min(tlo, r);
            thi = max(thi, r);
            return;
        }
        if (bin_d <= -(1 << 29)) return;          // invalid range: every tap is dropped
        for (int j = 0; j < kSincTaps; ++j) {
            const int b = bin_d - kSincTaps / 2 + j;
            if (b < 0 || b >= cb.nbins) continue;
            const float w = sinc[lut + j * kSincOvs];
#pragma unroll
            for (int o = 0; o < NOUT; ++o)
                if (o < cb.nout) cb.add_global(o, b, w * coef[o].re - 0.f * coef[o].im, w * coef[o].im + 0.f * coef[o].re);
        }
    }
};

// Tile end: out[b] = sum_{j, l} sinc[l + j ovs] H[b + taps/2 - j][l] over the touched rows of
// H, four lanes per output bin (two taps each), one compensated global add per bin.  Every
// thread calls it, after a barrier that completes H.
template <int NOUT>
OCS_D void hist_flush(const HistSmem<NOUT> &sm, int base, MixBins<NOUT> &cb) {
    int lo = kGridBins, hi = -1;
    for (int w = 0; w < kHistThreads / 32; ++w) {
        lo = min(lo, sm.range[w]);
        hi = max(hi, sm.range[8 + w]);
    }
    if (hi < lo) return;              // uniform: nothing landed in H
    const int nob = hi - lo + kSincTaps, items = nob * cb.nout * 4;
    // sums of every item of this thread first, then the returning adds, then their rounding
    // errors, so that the round trips to memory overlap
    constexpr int kPer = ((kGridBins + kSincTaps) * NOUT * 4 + kHistThreads - 1) / kHistThreads;
    float v[kPer], old[kPer];
    int at[kPer];                     // float offset in the raw row, -1: nothing to add
    const int q = threadIdx.x & 3;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        at[k] = -1;
        const int i = k * kHistThreads + threadIdx.x;
        if (k * kHistThreads >= items) continue;                  // uniform
        const int o = (i >> 2) / nob, m = (i >> 2) - o * nob;
        float sre = 0.f, sim = 0.f;
        if (i < items) {
            const float *hr = sm.h + (2 * o) * kGridBins * kGridL;
#pragma unroll
            for (int jj = 0; jj < kSincTaps / 4; ++jj) {
                const int j = q * (kSincTaps / 4) + jj, r = lo + m - j;
                if (r < lo || r > hi) continue;
                const float *w = sm.sinc + j * kGridL, *cr = hr + r * kGridL, *ci = cr + kGridBins * kGridL;
#pragma unroll
                for (int l = 0; l < kGridL; ++l) {
                    sre = fmaf(w[l], cr[l], sre);
                    sim = fmaf(w[l], ci[l], sim);
                }
            }
        }
        sre += __shfl_xor_sync(0xffffffffu, sre, 1);
        sim += __shfl_xor_sync(0xffffffffu, sim, 1);
        sre += __shfl_xor_sync(0xffffffffu, sre, 2);
        sim += __shfl_xor_sync(0xffffffffu, sim, 2);
        // lane 0 of the four adds the real part, lane 1 the imaginary part
        v[k] = q == 0 ? sre : sim;
        const int b = base + lo - kSincTaps / 2 + m;
        if (i < items && q < 2 && b >= 0 && b < cb.nbins && v[k] != 0.f) {
            at[k] = 2 * (o * cb.nbins + b) + q;
            old[k] = atomicAdd(cb.out + (long long)o * cb.out_stride + 2 * b + q, v[k]);
        }
    }
    if (!cb.lo_row) return;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        if (at[k] < 0) continue;
        const float e = two_sum_err(old[k], v[k], __fadd_rn(old[k], v[k]));
        if (e != 0.f) atomicAdd(cb.lo_row + at[k], e);
    }
}

// Read-only load at a 32-bit byte offset from a base shared by the warp.
template <class V> OCS_D V ld_at(const void *base, unsigned off) {
    return __ldg(reinterpret_cast<const V *>(static_cast<const char *>(base) + off));
}

// Staged inputs of one facet: fields, sqrt(RCS), scatterer-series values.
template <bool KODIS, int FAST> OCS_D void mix_load(const PulseArgs &a, unsigned off, long long plane, MixIn &in) {
    in.dx = ld_at<float>(a.dx_f, off);
    in.dy = ld_at<float>(a.dy_f, off);
    in.dz = ld_at<float>(a.dz_f, off);
    in.diffx = ld_at<float>(a.diffx, off);
    in.diffy = ld_at<float>(a.diffy, off);
    if (FAST || (KODIS && a.do_kodis)) {
        in.dxx = ld_at<float>(a.diffxx, off);
        in.dyy = ld_at<float>(a.diffyy, off);
        in.dxy = ld_at<float>(a.diffxy, off);
    }
    if (FAST || a.do_bragg) {
        const char *s = static_cast<const char *>(a.scat);
        in.sc[0][0] = ld_at<float>(s, off);
        in.sc[0][1] = ld_at<float>(s + plane, off);
        if (!FAST && a.npol == 2) {
            in.sc[1][0] = ld_at<float>(s + 2 * plane, off);
            in.sc[1][1] = ld_at<float>(s + 3 * plane, off);
        }
    }
}
OCS_D void mix_gather(const PulseArgs &a, int im, int ip, MixIn &in) {
    im += a.tmod_m;
    im = im >= a.n_m ? im - a.n_m : im;
    ip += a.tmod_p;
    ip = ip >= a.n_p ? ip - a.n_p : ip;
    in.cm = ld_at<float2>(a.s_m32, 8u * (unsigned)im);
    in.cp = ld_at<float2>(a.s_p32, 8u * (unsigned)ip);
}

// One tile of 128 columns x tile_rows rows, one column per thread, kHistStreams rows at a
// time; the inputs of the next row of a thread (and, one more row ahead, its scatterer
// indices) are loaded into registers while a row is processed.  Offsets are 32 bits
// (mixed_hist_ok bounds the surface and the series).
template <int NOUT, bool KODIS, int FAST>
OCS_D void mix_hist_tile(const PulseArgs &a, float *lo_row, int tile, int tile_rows, const HistSmem<NOUT> &sm,
                         double &spec_sum) {
    const int lane = threadIdx.x & 31;
    const int tiles_x = (a.nx + kMixCols - 1) / kMixCols;
    const int x0t = (tile % tiles_x) * kMixCols;
    const int x = x0t + threadIdx.x % kMixCols, stream = threadIdx.x / kMixCols;
    const int y0 = (tile / tiles_x) * tile_rows;
    const int nrows = min(tile_rows, a.ny - y0);
    constexpr int RT = mix_row_floats<NOUT>();
    const bool bragg = FAST || a.do_bragg;
    const bool busy = x < a.nx && stream < nrows;
    const long long plane = (long long)a.nx * a.ny * 4;
    // rows past the tile's last one repeat the thread's last row (loaded, not processed)
    const unsigned step = 4u * kHistStreams * (unsigned)a.nx;
    const unsigned off0 = 4u * ((unsigned)(y0 + stream) * (unsigned)a.nx + (unsigned)x);
    const unsigned last = off0 + (unsigned)((nrows - 1 - stream) / kHistStreams) * step;
    unsigned off = off0;
    // the first row's loads and the column constants, ahead of the barrier
    MixIn cur, nxt;
    MixCol col;
    int im = 0, ip = 0;
    if (busy) {
        if (bragg) { im = ld_at<int>(a.ind0_m, off); ip = ld_at<int>(a.ind0_p, off); }
        mix_load<KODIS, FAST>(a, off, plane, cur);
        col.init<KODIS, FAST>(a, x);
    }
    MixBins<NOUT> cb;
    cb.hi = cb.lo = nullptr;
    cb.cta_base = 0;
    cb.nout = FAST ? NOUT : a.nout;
    cb.nbins = a.nbins;
    cb.out = reinterpret_cast<float *>(a.raw) + 2 * ((long long)a.out0 * a.raw_out_stride + a.raw_row);
    cb.lo_row = lo_row ? lo_row + 2LL * a.out0 * a.nbins : nullptr;
    cb.out_stride = 2 * a.raw_out_stride;
    MixHist<NOUT, FAST> hist;
    hist.h = sm.h;
    hist.tlo = kGridBins;
    hist.thi = -1;
    {
        // H centred on the undisplaced bins of the tile's corners
        const double inv_sr0 = 1.0 / a.sr0;
        auto bin_at = [&](int xx, int yy) {
            const double az = (double)a.y[yy] - a.az_now;
            const double srg = a.sr_col[xx] + az * 0.5 * (az * inv_sr0);
            return (int)floor((srg - a.min_sr) * a.inv_binsize);
        };
        const int xb = min(x0t + kMixCols, a.nx) - 1;
        const int b0 = bin_at(x0t, y0), b1 = bin_at(xb, y0);
        const int b2 = bin_at(x0t, y0 + nrows - 1), b3 = bin_at(xb, y0 + nrows - 1);
        hist.base = (min(min(b0, b1), min(b2, b3)) + max(max(b0, b1), max(b2, b3)) - kGridBins) / 2;
    }
    if (busy && bragg) {
        mix_gather(a, im, ip, cur);
        const unsigned off2 = min(off + step, last);
        im = ld_at<int>(a.ind0_m, off2);
        ip = ld_at<int>(a.ind0_p, off2);
    }
    {
        eval_tile_rows<NOUT>(a, y0, nrows, sm.tmp, [&](int r, double az, double sin_az, double, double cos_azp, double sin_azp) {
            MixRow<NOUT>::store(sm.rt + r * RT, a, az, sin_az, cos_azp, sin_azp);
            double *ex = sm.exact + 4 * r;
            ex[0] = az; ex[1] = sin_az; ex[2] = cos_azp; ex[3] = sin_azp;
        });
        float4 *h4 = reinterpret_cast<float4 *>(sm.h);
        for (int i = threadIdx.x; i < NOUT * 2 * kGridBins * kGridL / 4; i += kHistThreads)
            h4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nrows * cb.nout; i += kHistThreads) {
        const int r = i / cb.nout, k = i - r * cb.nout;
        const c128 f = tile_factor<NOUT>(sm.tmp, r, k);
        sm.rt[r * RT + 6 + 2 * k] = (float)f.re;
        sm.rt[r * RT + 7 + 2 * k] = (float)f.im;
    }
    __syncthreads();
    if (busy) {
        const unsigned outs = mix_outs<NOUT>(a);
        for (int i = stream; i < nrows; i += kHistStreams) {
            off = min(off + step, last);
            mix_load<KODIS, FAST>(a, off, plane, nxt);
            if (bragg) {
                mix_gather(a, im, ip, nxt);
                const unsigned off2 = min(off + step, last);
                im = ld_at<int>(a.ind0_m, off2);
                ip = ld_at<int>(a.ind0_p, off2);
            }
            MixRow<NOUT> row;
            row.load(sm.rt + i * RT, sm.exact + 4 * i);
            int bin_d, lut;
            c64 coef[NOUT];
            mix_facet<NOUT, KODIS, FAST>(a, col, cur, row, outs, x, bin_d, lut, coef, spec_sum);
            hist.add(bin_d, lut, coef, a.sinc, cb);
            cur = nxt;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        hist.tlo = min(hist.tlo, __shfl_xor_sync(0xffffffffu, hist.tlo, o));
        hist.thi = max(hist.thi, __shfl_xor_sync(0xffffffffu, hist.thi, o));
    }
    if (lane == 0) {
        sm.range[threadIdx.x >> 5] = hist.tlo;
        sm.range[8 + (threadIdx.x >> 5)] = hist.thi;
    }
    __syncthreads();                      // H and the touched ranges are complete
    hist_flush<NOUT>(sm, hist.base, cb);
}

template <int NOUT> OCS_D void hist_init(const HistSmem<NOUT> &sm, const float *sinc) {
    for (int i = threadIdx.x; i < kSincTaps * kGridL; i += kHistThreads)
        sm.sinc[i] = sinc[i % kGridL + (i / kGridL) * kSincOvs];
}

// The last CTA of the launch to finish folds the compensation rows of the pass's outputs into
// their raw rows and clears them (every add of the launch has been made by then: each CTA
// counts itself in, past a fence, in the workspace header).  Every thread calls it.
OCS_D void fold_by_last(const PulseArgs &a, float *lo_row, int *shared_flag) {
    int *hdr = reinterpret_cast<int *>(reinterpret_cast<unsigned char *>(a.rowtab) + mix_hdr_offset(a.ny, a.nch));
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) *shared_flag = atomicAdd(hdr + 2, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!*shared_flag) return;
    __threadfence();
    float *raw = reinterpret_cast<float *>(a.raw);
    float2 *lo = reinterpret_cast<float2 *>(lo_row) + (long long)a.out0 * a.nbins;
    // batches of independent loads: this is the tail of the launch, one round trip per line
    constexpr int B = 8;
    const int n = a.nout * a.nbins;
    for (int i0 = threadIdx.x; i0 < n; i0 += B * kHistThreads) {
        float2 e[B], v[B];
        float2 *dst[B];
#pragma unroll
        for (int u = 0; u < B; ++u) {
            const int i = i0 + u * kHistThreads, k = i / a.nbins;
            dst[u] = reinterpret_cast<float2 *>(raw) + ((a.out0 + k) * a.raw_out_stride + a.raw_row + (i - k * a.nbins));
            e[u] = i < n ? __ldcg(lo + i) : make_float2(0.f, 0.f);
            v[u] = i < n ? __ldcg(dst[u]) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < B; ++u) {
            if (e[u].x == 0.f && e[u].y == 0.f) continue;
            *dst[u] = make_float2(v[u].x + e[u].x, v[u].y + e[u].y);
            lo[i0 + u * kHistThreads] = make_float2(0.f, 0.f);
        }
    }
    if (threadIdx.x == 0) hdr[2] = 0;
}

// Three resident CTAs, two and three for one, two, three and four outputs: 2048^2 80, 92, 128, 110
// and 72, 83, 120, 110 us; 512^2 13.6, 15.6, 18.7, 18.5 and 14.5, 16.1, 20.1, 20.3.
template <int NOUT, bool KODIS, int FAST>
__global__ void __launch_bounds__(kHistThreads, 3)
pulse_mixed_hist_kernel(const __grid_constant__ PulseArgs a, float *lo_row) {
    extern __shared__ __align__(16) unsigned char hist_raw[];
    const HistSmem<NOUT> sm = hist_smem<NOUT>(hist_raw, kPulseRows);
    grid_wait();
    hist_init<NOUT>(sm, a.sinc);
    double spec_sum = 0.0;
    mix_hist_tile<NOUT, KODIS, FAST>(a, lo_row, blockIdx.x, a.tile_rows, sm, spec_sum);
    if (a.out0 == 0 && KODIS) block_atomic_sum(spec_sum, &a.nrcs_spec[a.az_step], sm.sred);
    if (lo_row) fold_by_last(a, lo_row, sm.range);
}

// Rows of a tile whose cells of H sum at most kCellFacets facets each, with 20 LUT cells per bin
// that the tile's columns span (waves only spread them further).  A cell's float32 sum rounds once
// per facet and the convolution 44 times more; the register windows round 64 times per tile column
// and 32 times across a warp before their first compensated add, so 48 facets keep the grid's
// bound below theirs (92 and 96 roundings).  Facets of 1 m at 35 degrees in 2.7 m bins have 202
// rows, of 0.5 m at 12 degrees 36.  Measured on a flat sea of 2048^2 equal facets, largest error of
// a bin, windows / grid with tiles of 38 rows / grid with these: facets of 1 m 1.4e-7 / 1.2e-7 /
// 1.3e-7, 0.05 m 1.1e-7 / 1.6e-7 / 0.7e-7, 0.02 m 0.6e-7 / 2.7e-7 / 0.6e-7.
constexpr int kCellFacets = 48;
inline int mixed_hist_rows(double span) {
    const double rows = kCellFacets * kSincOvs * span / kMixCols;
    return rows < kPulseRowsMax ? (int)rows : kPulseRowsMax;
}

// Whether the fine-grid form takes a pulse: its byte offsets into the planes (4 bytes a facet) and
// into the scatterer series (8 bytes an entry; n_series: the longer one's entries) are 32 bits,
// its cells allow tiles of `least` rows, and H leaves the waves kGridMargin metres of range on each
// side of a tile's columns (grid_holds_tile's six bins are more from 0.42 m a bin up): a facet
// outside H costs returning adds of every tap to memory.  1024 x 512 facets, two channels, windows
// and grid: 0.11 m in bins of 0.23 m (1.4 m left) in seas of 3 m significant height 58 and 84 us,
// 0.08 m (2.5 m) 37 and 20; 0.03 m in bins of 0.11 m (1.6 m) at 6 m 126 and 160; 0.22 m in bins of
// 0.45 m (2.8 m) 106 and 85.  The float64 grid, whose adds return nothing, needs no such bound: it
// is level or faster there (1.6 m left at 6 m 136 and 94; at 10 m, of 22 bins' standard deviation,
// it is not, 161 and 461).
constexpr double kGridMargin = 2.5;
inline bool mixed_hist_ok(int nx, int ny, long long n_series, double span, double binsize, int least) {
    return (long long)nx * ny < (1LL << 30) && n_series < (1LL << 29) && grid_holds_tile(span) &&
           (kGridBins - span) * binsize >= 2.0 * kGridMargin && mixed_hist_rows(span) >= (ny < least ? ny : least);
}
// The rows that a single scene's pulse asks for: those of its tiles on 148 SMs, up to 28.  Shorter
// tiles than its own cost a pulse their rows' set-up and flush, and a warp's adds to few cells
// wait for one another: 2048^2 (38 rows of their own), one channel, facets of 1 m 72 us, 0.1 m (20
// rows) 94 and windows 90, two channels 109 and 97; 0.05 m (10 rows) 127 and 90; 1024 x 512 (10
// rows of their own), 0.05 m, 20 and 32.
inline int hist_least_rows(int nx, int ny) {
    const int own = tile_rows_for(nx, ny, kMixCols, 3 * 148, kHistStreams);
    return own < 28 ? own : 28;
}

// Launches of pulse_split.cu: the output group [a.out0, a.out0 + a.nout) of one pulse (maps:
// the inputs' tensor maps, used by the register-window form only; hist_rows: the tallest tiles of
// the fine grid, 0 for the register windows), and one batch class.
int split_hist_rows(const PulseArgs &a);
int launch_pulse_split(const PulseArgs &a, const MixMaps &maps, float *lo_row, int hist_rows, cudaStream_t st);
int batch_pulse_split(const BatchRef &b, int kind, int width, int grid, cudaStream_t st);

}  // namespace ocs
