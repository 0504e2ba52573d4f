// Float64 pulse of SAR scenes with Kodis specular and / or Romeiser Bragg scattering: the
// drop-in form of the azimuth loop's body (oceansar/radarsim/sar_raw_nompi.py:349-535), every
// operation in float64 in the reference's order where it decides a discrete outcome (slant
// range, range bin, LUT index, specular facet window), through a fine-grid accumulation.
//
// What bounds it: latency.  The register-window kernel (pulse_core.cuh) holds 12 bins x 2
// outputs in 96 registers of its 238, so 8 warps fit an SM (issue active 27%), four outputs take
// two passes that both evaluate the facet physics, and its tile-end flush adds every lane's
// window to the same few shared bins one after the other.  Here a facet adds its coefficient
// once per output into a shared (bin, LUT index) grid H, convolved with the pulse at the tile's
// end: no windows, up to four outputs in one pass, 16 warps per SM, tiles as short as a
// small surface needs to fill the GPU.
// Measured per ordinary pulse: 1024^2 facets, two channels x two polarisations 2 x 97 -> 50 us;
// 512^2, one channel 30 -> 10.4 us.
//
// The two Bragg phases -2 k0 r -/+ cap of a facet share the sine and cosine of 2 k0 r: with
// d = fl(s - c) and e = (s - c) - d (exact, TwoSum), exp(i d) = exp(i s) exp(-i c) exp(-i e),
// and |e| is at most half an ulp of the phase, so exp(-i e) = 1 - i e to float64 accuracy.
// The rounding of the phase that the reference makes is thereby kept.
#pragma once
#include "pulse_core.cuh"

namespace ocs {

constexpr int kF64Threads = 256;    // 128 columns x 2 rows
constexpr int kF64Streams = kF64Threads / kPulseCols;

template <int NOUT> struct F64Smem {
    double *sred;                   // block reduction scratch [32]
    double *sinc;                   // [taps][kGridL]
    double *h;                      // [NOUT][re, im][kGridBins][kGridL]
    double *rt;                     // rows of the tile [rows][4 + 2 NOUT]
    double *tmp;                    // eval_tile_rows scratch [rows][2 + 2 NOUT]
    int *range;                     // touched rows of H of each warp [2][8]
};
template <int NOUT> OCS_HD constexpr int f64_rt() { return 4 + 2 * NOUT; }
template <int NOUT> OCS_HD constexpr size_t f64_smem_bytes(int rows_cap) {
    return (32 + kSincTaps * kGridL + (size_t)NOUT * 2 * kGridBins * kGridL + (size_t)rows_cap * (f64_rt<NOUT>() + 2 + 2 * NOUT)) * 8 +
           16 * 4;
}
template <int NOUT> OCS_D F64Smem<NOUT> f64_smem(unsigned char *smem, int rows_cap) {
    F64Smem<NOUT> sm;
    sm.sred = reinterpret_cast<double *>(smem);
    sm.sinc = sm.sred + 32;
    sm.h = sm.sinc + kSincTaps * kGridL;
    sm.rt = sm.h + NOUT * 2 * kGridBins * kGridL;
    sm.tmp = sm.rt + rows_cap * f64_rt<NOUT>();
    sm.range = reinterpret_cast<int *>(sm.tmp + rows_cap * (2 + 2 * NOUT));
    return sm;
}

// Read-only load at a 32-bit byte offset from a base shared by the warp.
template <class V> OCS_D V f64_at(const void *base, unsigned off) {
    return __ldg(reinterpret_cast<const V *>(static_cast<const char *>(base) + off));
}

// Inputs of one facet: fields, sqrt(RCS) of both lines per polarisation, scatterer values.
template <int NPOL> struct F64In {
    float dx, dy, dz, diffx, diffy, dxx, dyy, dxy;
    double sc[2 * NPOL];
    double2 cm, cp;
    OCS_D void load(const PulseArgs &a, unsigned off, long long plane8) {
        dx = f64_at<float>(a.dx_f, off);
        dy = f64_at<float>(a.dy_f, off);
        dz = f64_at<float>(a.dz_f, off);
        if (a.do_kodis) {
            diffx = f64_at<float>(a.diffx, off);
            diffy = f64_at<float>(a.diffy, off);
            dxx = f64_at<float>(a.diffxx, off);
            dyy = f64_at<float>(a.diffyy, off);
            dxy = f64_at<float>(a.diffxy, off);
        }
        if (a.do_bragg) {
            const char *s = static_cast<const char *>(a.scat);
#pragma unroll
            for (int k = 0; k < 2 * NPOL; ++k) sc[k] = f64_at<double>(s + k * plane8, 2u * off);
        }
    }
    OCS_D void gather(const PulseArgs &a, int im, int ip) {
        im += a.tmod_m;
        im = im >= a.n_m ? im - a.n_m : im;
        ip += a.tmod_p;
        ip = ip >= a.n_p ? ip - a.n_p : ip;
        cm = __ldg(reinterpret_cast<const double2 *>(a.s_m) + im);
        cp = __ldg(reinterpret_cast<const double2 *>(a.s_p) + ip);
    }
};

// exp(i fl(s + c)) from the unit vectors of s and c.
OCS_D c128 phase_sum(double s, double c, c128 es, c128 ec) {
    const double d = dadd(s, c), bp = dsub(d, s);
    const double e = dadd(dsub(s, dsub(d, bp)), dsub(c, bp));          // (s + c) - d, exact
    const c128 v = cmul(es, ec);
    return {fma(e, v.im, v.re), fma(-e, v.re, v.im)};                  // times 1 - i e
}

// Out-of-grid or non-finite facet: per-tap global adds, exactly its own taps.
template <int NOUT>
OCS_D void f64_direct(const PulseArgs &a, int bin_d, int lut, const c128 (&coef)[NOUT]) {
    double *out = reinterpret_cast<double *>(a.raw) + 2 * ((long long)a.out0 * a.raw_out_stride + a.raw_row);
    for (int j = 0; j < kSincTaps; ++j) {
        const int b = bin_d - kSincTaps / 2 + j;
        if (b < 0 || b >= a.nbins) continue;
        const double w = (double)a.sinc[lut + j * kSincOvs];
#pragma unroll
        for (int o = 0; o < NOUT; ++o) {
            if (o >= a.nout) continue;
            double *d = out + 2 * (o * a.raw_out_stride + b);
            atomicAdd(d, w * coef[o].re - 0.0 * coef[o].im);
            atomicAdd(d + 1, w * coef[o].im + 0.0 * coef[o].re);
        }
    }
}

// One tile of 128 columns x tile_rows rows, one column per thread, kF64Streams rows at a time;
// the next row's inputs (and, one more row ahead, its scatterer indices) are loaded into
// registers while a row is processed.
template <int NOUT, int NPOL, bool XTI>
OCS_D void f64_tile(const PulseArgs &a, int tile, int tile_rows, const F64Smem<NOUT> &sm, double &spec_sum) {
    constexpr int RT = f64_rt<NOUT>();
    const int tiles_x = (a.nx + kPulseCols - 1) / kPulseCols;
    const int x0t = (tile % tiles_x) * kPulseCols;
    const int x = x0t + threadIdx.x % kPulseCols, stream = threadIdx.x / kPulseCols;
    const int y0 = (tile / tiles_x) * tile_rows;
    const int nrows = min(tile_rows, a.ny - y0);
    const bool busy = x < a.nx && stream < nrows;
    const long long plane8 = (long long)a.nx * a.ny * 8;
    // rows past the tile's last one repeat the thread's last row (loaded, not processed)
    const unsigned step = 4u * kF64Streams * (unsigned)a.nx;
    unsigned off = 4u * ((unsigned)(y0 + stream) * (unsigned)a.nx + (unsigned)x);
    const unsigned last = off + (unsigned)((nrows - 1 - stream) / kF64Streams) * step;
    F64In<NPOL> cur, nxt;
    int im = 0, ip = 0;
    if (busy) {
        if (a.do_bragg) { im = f64_at<int>(a.ind0_m, off); ip = f64_at<int>(a.ind0_p, off); }
        cur.load(a, off, plane8);
    }
    // channel and polarisation of every output of the pass
    int och[NOUT], opol[NOUT];
#pragma unroll
    for (int k = 0; k < NOUT; ++k) {
        const int o = min(a.out0 + k, a.npol * a.nch - 1);
        opol[k] = NPOL == 1 ? 0 : o / a.nch;
        och[k] = o - opol[k] * a.nch;
    }
    // rows: az, sin_az, cos and sin of the azimuth angle, then the outputs' factors
    eval_tile_rows<NOUT>(a, y0, nrows, sm.tmp, [&](int r, double az, double sin_az, double, double cos_azp, double sin_azp) {
        double *row = sm.rt + r * RT;
        row[0] = az; row[1] = sin_az; row[2] = cos_azp; row[3] = sin_azp;
    });
    int base;
    {
        // H centred on the undisplaced bins of the tile's corners
        const double inv_sr0 = 1.0 / a.sr0;
        auto bin_at = [&](int xx, int yy) {
            const double az = (double)a.y[yy] - a.az_now;
            const double srg = a.sr_col[xx] + az * 0.5 * (az * inv_sr0);
            return (int)floor((srg - a.min_sr) * a.inv_binsize);
        };
        const int xb = min(x0t + kPulseCols, a.nx) - 1;
        const int b0 = bin_at(x0t, y0), b1 = bin_at(xb, y0);
        const int b2 = bin_at(x0t, y0 + nrows - 1), b3 = bin_at(xb, y0 + nrows - 1);
        base = (min(min(b0, b1), min(b2, b3)) + max(max(b0, b1), max(b2, b3)) - kGridBins) / 2;
    }
    for (int i = threadIdx.x; i < NOUT * 2 * kGridBins * kGridL; i += kF64Threads) sm.h[i] = 0.0;
    int tlo = kGridBins, thi = -1;
    double sr_c = 0.0, sin_i = 0.0, cos_i = 0.0, tan_i = 0.0, cap = 0.0, dinc0 = 0.0;
    c128 ecap = {1.0, 0.0};
    if (busy) {
        sr_c = a.sr_col[x];
        sin_i = a.sin_inc[x];
        cos_i = a.cos_inc[x];
        if (a.do_kodis) tan_i = a.tan_inc[x];
        if (XTI) dinc0 = a.inc[x] - a.inc_angle;
        if (a.do_bragg) {
            cap = ((2.0 * a.k0) * a.t_step) * a.c_b[x] * (double)(a.az_step + 1);
            ecap = cexpi(cap);
            cur.gather(a, im, ip);
            const unsigned off2 = min(off + step, last);
            im = f64_at<int>(a.ind0_m, off2);
            ip = f64_at<int>(a.ind0_p, off2);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nrows * a.nout; i += kF64Threads) {
        const int r = i / a.nout, k = i - r * a.nout;
        const c128 f = tile_factor<NOUT>(sm.tmp, r, k);
        sm.rt[r * RT + 4 + 2 * k] = f.re;
        sm.rt[r * RT + 5 + 2 * k] = f.im;
    }
    __syncthreads();
    if (busy) {
        const double two_k0 = 2.0 * a.k0;
        for (int i = stream; i < nrows; i += kF64Streams) {
            off = min(off + step, last);
            nxt.load(a, off, plane8);
            if (a.do_bragg) {
                nxt.gather(a, im, ip);
                const unsigned off2 = min(off + step, last);
                im = f64_at<int>(a.ind0_m, off2);
                ip = f64_at<int>(a.ind0_p, off2);
            }
            const double *rt = sm.rt + i * RT;
            const double sin_az = rt[1];
            // slant range: sr - cos_inc*Dz + az/2*sin_az + Dx*sin_inc + Dy*sin_az, left to
            // right, no fused multiply-adds (bit-identical with numpy)
            double srs = dsub(sr_c, dmul(cos_i, (double)cur.dz));
            srs = dadd(srs, dmul(rt[0] * 0.5, sin_az));
            srs = dadd(srs, dmul((double)cur.dx, sin_i));
            srs = dadd(srs, dmul((double)cur.dy, sin_az));
            int bin_d, lut;
            bin_lut_magic(div_by(dsub(srs, a.min_sr), a.binsize, a.inv_binsize), (double)kSincOvs, bin_d, lut);
            c128 scene[NPOL];
#pragma unroll
            for (int p = 0; p < NPOL; ++p) scene[p] = {0.0, 0.0};
            if (a.do_kodis) {
                const c128 e = kodis_facet<double>(a.kodis, srs, sin_i, cos_i, tan_i, rt[2], rt[3], cur.diffx,
                                                   cur.diffy, cur.dxx, cur.dyy, cur.dxy);
                const double s4 = 3.5449077018110318;                 // sqrt(4 pi)
                const c128 es = {e.re * s4, e.im * s4};
                spec_sum += es.re * es.re + es.im * es.im;
#pragma unroll
                for (int p = 0; p < NPOL; ++p) scene[p] = es;
            }
            if (a.do_bragg) {
                // Bragg phases: -2 k0 r -/+ 2 k0 t_step c_b (az_step + 1)
                const double surf = (-two_k0) * srs;
                const c128 es = cexpi(surf);
                const c128 e0 = cmul(phase_sum(surf, -cap, es, {ecap.re, -ecap.im}), c128{cur.cm.x, cur.cm.y});
                const c128 e1 = cmul(phase_sum(surf, cap, es, ecap), c128{cur.cp.x, cur.cp.y});
#pragma unroll
                for (int p = 0; p < NPOL; ++p) {
                    scene[p].re += cur.sc[2 * p] * e0.re + cur.sc[2 * p + 1] * e1.re;
                    scene[p].im += cur.sc[2 * p] * e0.im + cur.sc[2 * p + 1] * e1.im;
                }
            }
            // channels of this pass: antenna pattern x ATI phase (per row) x XTI phase
            c128 coef[NOUT];
            double wave_dinc = 0.0, sum = 0.0;
            if (XTI) wave_dinc = ((double)cur.dz * sin_i + (double)cur.dx * sin_i) / a.sr0;
#pragma unroll
            for (int k = 0; k < NOUT; ++k) {
                c128 v = scene[0];
                if (NPOL == 2 && opol[k]) v = scene[NPOL - 1];
                v = cmul(v, c128{rt[4 + 2 * k], rt[5 + 2 * k]});
                if (XTI && a.b_xti[och[k]] != 0.0) v = cmul(v, cexpi((-a.k0 * a.b_xti[och[k]]) * (dinc0 + wave_dinc)));
                coef[k] = v;
                if (k < a.nout) sum += v.re + v.im;
            }
            const int r = bin_d - base;
            if ((unsigned)r < (unsigned)kGridBins && isfinite(sum)) {
                double *h = sm.h + r * kGridL + lut;
#pragma unroll
                for (int k = 0; k < NOUT; ++k) {
                    if (k < a.nout) {
                        atomicAdd(h + (2 * k) * kGridBins * kGridL, coef[k].re);
                        atomicAdd(h + (2 * k + 1) * kGridBins * kGridL, coef[k].im);
                    }
                }
                tlo = min(tlo, r);
                thi = max(thi, r);
            } else if (bin_d > -(1 << 29)) {
                f64_direct<NOUT>(a, bin_d, lut, coef);
            }
            cur = nxt;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tlo = min(tlo, __shfl_xor_sync(0xffffffffu, tlo, o));
        thi = max(thi, __shfl_xor_sync(0xffffffffu, thi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        sm.range[threadIdx.x >> 5] = tlo;
        sm.range[8 + (threadIdx.x >> 5)] = thi;
    }
    __syncthreads();                      // H and the touched ranges are complete
    int lo = kGridBins, hi = -1;
    for (int w = 0; w < kF64Threads / 32; ++w) {
        lo = min(lo, sm.range[w]);
        hi = max(hi, sm.range[8 + w]);
    }
    if (hi < lo) return;                  // uniform: nothing landed in H
    // out[b] = sum_{j, l} sinc[l + j ovs] H[b + taps/2 - j][l] over the touched rows of H: four
    // lanes per output bin, two taps each; lane 0 adds the real part, lane 1 the imaginary
    const int nob = hi - lo + kSincTaps, items = nob * a.nout * 4;
    double *out = reinterpret_cast<double *>(a.raw) + 2 * ((long long)a.out0 * a.raw_out_stride + a.raw_row);
    const int q = threadIdx.x & 3;
    for (int i0 = 0; i0 < items; i0 += kF64Threads) {
        const int i = i0 + threadIdx.x;
        const int o = (i >> 2) / nob, m = (i >> 2) - o * nob;
        double sre = 0.0, sim = 0.0;
        if (i < items) {
            const double *hr = sm.h + (2 * o) * kGridBins * kGridL;
#pragma unroll
            for (int jj = 0; jj < kSincTaps / 4; ++jj) {
                const int j = q * (kSincTaps / 4) + jj, r = lo + m - j;
                if (r < lo || r > hi) continue;
                const double *w = sm.sinc + j * kGridL, *cr = hr + r * kGridL, *ci = cr + kGridBins * kGridL;
                for (int l = 0; l < kGridL; ++l) {
                    sre = fma(w[l], cr[l], sre);
                    sim = fma(w[l], ci[l], sim);
                }
            }
        }
        sre += __shfl_xor_sync(0xffffffffu, sre, 1);
        sim += __shfl_xor_sync(0xffffffffu, sim, 1);
        sre += __shfl_xor_sync(0xffffffffu, sre, 2);
        sim += __shfl_xor_sync(0xffffffffu, sim, 2);
        const int b = base + lo - kSincTaps / 2 + m;
        const double v = q == 0 ? sre : sim;
        if (i < items && q < 2 && b >= 0 && b < a.nbins && v != 0.0)
            atomicAdd(out + 2 * (o * a.raw_out_stride + b) + q, v);
    }
}

template <int NOUT> OCS_D void f64_init(const F64Smem<NOUT> &sm, const float *sinc) {
    for (int i = threadIdx.x; i < kSincTaps * kGridL; i += kF64Threads)
        sm.sinc[i] = (double)sinc[i % kGridL + (i / kGridL) * kSincOvs];
}

// Whether the kernel takes a pulse: a SAR pulse whose 128-column tiles fit the grid and span half
// a bin (ten cells) or more, and whose float64 planes 32-bit offsets can address.  A warp's adds to
// fewer cells wait for one another: 2048^2 facets in bins of 2.7 m, windows and grid, of 0.03 m 280
// and 142 us (four outputs 688 and 356), of 0.01 m (six cells) 287 and 255 (713 and 789), of 0.003 m
// 289 and 505 (715 and 1077).
inline bool f64_grid_ok(int nx, int ny, double span) {
    return (long long)nx * ny < (1LL << 29) && grid_holds_tile(span) && span >= 0.5;
}
int launch_pulse_f64(PulseArgs a, cudaStream_t st);
int batch_pulse_f64(const BatchRef &b, int width, int grid, cudaStream_t st);

}  // namespace ocs
