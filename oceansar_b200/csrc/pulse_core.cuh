// One radar pulse of the raw-data generator on sm_100a: the body of the azimuth loop of
// sar_raw (oceansar/radarsim/sar_raw_nompi.py:349-535) after the surface update, fused
// into one kernel per pulse so that no per-facet intermediate ever reaches HBM:
//
//   slant range of every facet (:366-369), Kodis specular field (:392-400),
//   Romeiser Bragg RCS refreshed every ocean_dt (:431-458, stored as sqrt(RCS) between
//   refreshes), Bragg phases + random sub-grid scatterers (:470-480), antenna pattern and
//   per-channel ATI / XTI phases (:485-495), and the range-profile accumulation
//   (range_profile.py:83-116) through the register-window engine of accum.cuh.
//
// Layout: a CTA owns BX consecutive ground-range columns (one per thread) and a strip of
// rows; each thread walks its column down the strip, so a warp reads 32 consecutive
// float32 of every field (coalesced) and its range bins drift slowly, keeping the
// register windows warm.  Per-row quantities (azimuth, antenna pattern, ATI phase) are
// computed once per CTA into shared memory.
//
// Scatterometer mode (MODE = kModeSca, the DopSCA generator, oceansar/dopscasim/dopsca_raw.py:
// 343-520): the columns are N_repeat_x range blocks side by side, each reading the same
// surface (field column = column mod field_nx) with its rows rolled by the integer azimuth
// shift (field row = (row + roll) mod ny); the scene is scaled by (sr0 / (sr0 + r))^2, the
// Bragg RCS is evaluated on every launch, the Bragg phase advances with the sub-pulse time
// cap_t, the range bins see the sub-pulse delay sr_bin_off, and the NRCS sums are kept per
// range block.
//
// SKIM mode (MODE & kModeSkim, the SKIM generator, oceansar/radarsim/skim_raw.py:465-689):
// sin_az = az / sr per facet (absolute slant range of the column), the two-way antenna
// pattern evaluated per facet, 10-tap pulse, and the facets of every ny_integ rows
// accumulated into their own output row (the two-scale Doppler's range-only profiles
// summed over ny_integ rows; ny_integ = ny gives the single-row form).
//
// Precision forms (template T):
//   double -- the drop-in: every operation in float64 in the reference's order; slant
//             range and the bin / LUT indices bit-identical to numpy.
//   float  -- mixed: slant range, bin / LUT indices and the 2 k0 r phase reduction in
//             float64, everything else (NRCS, scene, accumulation) in float32.
#pragma once
#include <string.h>

#include "accum.cuh"
#include "batch.cuh"
#include "physics.cuh"

namespace ocs {

constexpr int kPulseCols = 128;     // columns (threads) per CTA
constexpr int kPulseRows = 64;      // rows per tile (single-scene launches)
constexpr int kPulseRowsMax = 128;  // largest rows per tile (shared row tables)
constexpr int kMaxCh = 8;
constexpr int kPulseNbw = 160;      // CTA shared bin window
constexpr int kGridBins = 48;       // range bins of a fine-grid tile
constexpr int kGridL = kSincOvs + 1;   // LUT positions of a bin

// Kernel modes (bits): Kirchhoff specular, scatterometer (DopSCA), SKIM; SKIM combines with
// the Kirchhoff specular term (kModeSkim | kModeKa).
enum { kModeStd = 0, kModeKa = 1, kModeSca = 2, kModeSkim = 4 };
constexpr int kSkimTaps = 10;       // n_sinc_samples of the SKIM generator (skim_raw.py:164)
template <int MODE> __host__ __device__ constexpr int mode_taps() { return (MODE & kModeSkim) ? kSkimTaps : kSincTaps; }

struct PulseArgs {
    int nx, ny, npol, nch;
    int out0, nout;                         // outputs [out0, out0+nout) of npol*nch, o = pol*nch + ch
    const float *dx_f, *dy_f, *dz_f, *diffx, *diffy, *diffxx, *diffyy, *diffxy, *hmtf;
    const float *y;                         // [ny] float32 azimuth coordinates
    const double *sr_col, *sin_inc, *cos_inc, *tan_inc, *inc, *c_b;   // [nx]
    double inc_angle, sr0, gr0, k0, az_now, min_sr, binsize, inv_binsize, t_step;
    int any_xti;
    int az_step;
    long long tind;                         // int(t_now * prf)
    double ltx_over_l, lrx_over_l;          // antenna length / wavelength
    double b_ati[kMaxCh], b_xti[kMaxCh];
    int do_kodis, do_bragg, refresh, use_hmtf;
    KodisParams kodis;
    RomeiserParams rom;
    void *scat;                             // [npol][2][ny][nx] sqrt(RCS) (T)
    const double *s_m, *s_p;                // complex128 random-scatterer series
    const float *s_m32, *s_p32;             // complex64 copies (mixed form), or null
    int n_m, n_p;
    int tmod_m, tmod_p;                     // int(t_now * prf) mod n_m, n_p
    const int *ind0_m, *ind0_p;             // [ny][nx]
    const float *sinc;                      // [8*20 + 1]
    double *rowtab;                         // per-pulse row table, see pulse_rows_kernel
    void *raw;                              // [npol*nch][az_steps][rg_samp] complex T
    long long raw_out_stride, raw_row;      // elements between outputs, offset of this pulse row
    int nbins;
    double *nrcs_spec;                      // [az_steps]  sum |E_spec|^2
    double *nrcs_bragg;                     // [npol][az_steps] sum RCS (refresh pulses)
    int az_steps;
    int tile_rows;                          // rows per tile of a single-scene launch
    int spec_mode;                          // 0 Kodis, 1 Kirchhoff facet approach, 2 stationary phase
    const float *x_f;                       // [nx] facet x positions (Kirchhoff)
    KaParams ka;
    const void *lut;                        // Romeiser LUT [npol][2][naz][ndy][ndx] (T), or null
    int lut_naz, lut_ndy, lut_ndx;
    double lut_az0, lut_daz, lut_dy0, lut_ddy, lut_dx0, lut_ddx;
    int sca;                                // scatterometer mode (see the file comment)
    int fnx, roll;                          // field columns, azimuth roll of the field rows
    double sr_bin_off, cap_t;               // sub-pulse range delay, Bragg phase time
    int nblk, nrcs_row, nrcs_rows;          // range blocks; NRCS row of this call, rows in all
    int az_f32;                             // azimuth y - az_now rounded to float32 (see pulse_row)
    int skim, ny_integ, s_int;              // SKIM mode: output row per ny_integ facet rows
    int skim_az2, skim_rcm;                 // SKIM: az/2 sin_az in the phase range / in the bins only
    double atx, arx;                        // SKIM: antenna lengths / wavelength (tx, rx)
    int pt_mode, pt_x, pt_y;                // SKIM calibration target: 0 none, 1 floating, 2 fixed
    double pt_amp;
    long long lut_block;                    // scatterometer LUT: elements between block tables
    // float32 constants of the split-range form: 1 / binsize, 2 k0 (high and low part), facet
    // half sizes, 1 / sr0, R / 2, and -k0 b_xti of every channel
    float f_inv_bs, f_khi, f_klo, f_hdx, f_hdy, f_inv_sr0, f_hr, f_hi, f_kxti[kMaxCh];
};

// Kirchhoff specular term of one facet and polarisation code pc (0 = hh, 1 = vv),
// sar_raw_nompi.py:402-426: exp(-1j (2 k0 r)) (4 pi)^1.5 RCSKA.field(1, 1, ...).  Only the
// Kirchhoff instantiations of the pulse kernel (MODE = kModeKa) contain it.
OCS_D c128 ka_specular(const KaParams &kp, int pc, double srs, double x, double y, double st,
                                         double ct, double tt, double sp, double cp, float dz, float dx, float dy,
                                         float dxx, float dyy, float dxy) {
    const c128 e = ka_facet(kp, pc, pc, x, y, st, ct, tt, sp, cp, dz, dx, dy, dxx, dyy, dxy);
    const c128 ph = cexpi(-dmul(2.0 * kp.k0, srs));
    const double s15 = 44.54662397465366;                // (4 pi)^1.5
    return cmul128(cmulr(ph, s15), e);
}

// LUT mode of the Romeiser model (romeiser97.py:109-134): RCS of both Bragg lines of
// polarisation p at (azimuth index of the row, clamped slope indices of the facet).
// Indices round half to even from float64 differences and divisions, as numpy does.
template <typename T>
OCS_D void romeiser_lut(const PulseArgs &a, int az_ind, float diffx, float diffy, int p, T (&r)[2],
                        long long table = 0) {
    int iy = (int)rint(ddiv(dsub((double)diffy, a.lut_dy0), a.lut_ddy));
    int ix = (int)rint(ddiv(dsub((double)diffx, a.lut_dx0), a.lut_ddx));
    iy = iy > 0 ? (iy < a.lut_ndy ? iy : a.lut_ndy - 1) : 0;
    ix = ix > 0 ? (ix < a.lut_ndx ? ix : a.lut_ndx - 1) : 0;
    const T *lut = static_cast<const T *>(a.lut) + table;
    const long long plane = (long long)a.lut_naz * a.lut_ndy * a.lut_ndx;
    const long long off = ((long long)az_ind * a.lut_ndy + iy) * a.lut_ndx + ix;
    r[0] = lut[(2LL * p) * plane + off];
    r[1] = lut[(2LL * p + 1) * plane + off];
}

// Azimuth index of a row's ground-projected azimuth angle (negative: from the end, as numpy
// indexing takes it; out-of-table rows are rejected by the host before launch, and are
// clamped here so that no access leaves the table).
OCS_D int lut_az_index(const PulseArgs &a, double azp) {
    int i = (int)rint(ddiv(dsub(azp, a.lut_az0), a.lut_daz));
    if (i < 0) i += a.lut_naz;
    return i < 0 ? 0 : (i >= a.lut_naz ? a.lut_naz - 1 : i);
}

// Asynchronous global -> shared copies (cp.async): each thread copies the words it will
// read itself, so a cp.async.wait_group by that thread is all the ordering needed.
OCS_D void cp_async(void *dst, const void *src, int bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (bytes == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
    else if (bytes == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
OCS_D void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> OCS_D void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Staging of the per-facet inputs in shared memory: stage_rows rows of every input array
// ([8] float32 fields, [4] sqrt(RCS) of type T, [2] int32 scatterer offsets, kPulseCols
// columns each) in a ring of stage_rows slots, and two slots of the
// gathered scatterer-series values (complex128 of both Bragg lines), filled one row ahead.
// Ring slots: the mixed form keeps two rows in flight while it processes one (four
// slots); the float64 form, limited to two CTAs per SM by its registers, one (three slots,
// measured faster there).
template <typename T> OCS_HD constexpr int stage_rows() { return sizeof(T) == 4 ? 4 : 3; }
template <typename T> OCS_HD constexpr size_t stage_slot_bytes() {
    return (8 * 4 + 4 * sizeof(T) + 2 * 4) * (size_t)kPulseCols;
}
template <typename T> OCS_HD constexpr size_t stage_bytes() {
    return stage_rows<T>() * stage_slot_bytes<T>() + 2 * 2 * 16 * (size_t)kPulseCols + 16;
}

template <typename T> struct Stage {
    unsigned char *base;          // 16-byte aligned
    OCS_D float *f(int slot, int k) const {
        return reinterpret_cast<float *>(base + slot * stage_slot_bytes<T>()) + k * kPulseCols + threadIdx.x;
    }
    OCS_D T *scat(int slot, int k) const {
        return reinterpret_cast<T *>(base + slot * stage_slot_bytes<T>() + 32 * kPulseCols) + k * kPulseCols +
               threadIdx.x;
    }
    OCS_D int *ind(int slot, int k) const {
        return reinterpret_cast<int *>(base + slot * stage_slot_bytes<T>() + (32 + 4 * sizeof(T)) * kPulseCols) +
               k * kPulseCols + threadIdx.x;
    }
    OCS_D double2 *gather(int g, int k) const {
        return reinterpret_cast<double2 *>(base + stage_rows<T>() * stage_slot_bytes<T>()) + (2 * g + k) * kPulseCols +
               threadIdx.x;
    }
};

// Inputs of one facet.
template <typename T> struct FacetIn {
    float dx, dy, dz, diffx, diffy, diffxx, diffyy, diffxy;
    T scat[2][2];
    // start the copies of facet idx's inputs into stage slot `slot`
    // (fidx: index into the surface fields; idx: into the per-facet scatterer arrays)
    template <typename A>
    static OCS_D void issue(const A &a, const Stage<T> &st, int slot, long long idx, long long npix,
                            const T *scat_buf, bool load_scat, long long fidx) {
        cp_async(st.f(slot, 0), a.dx_f + fidx, 4);
        cp_async(st.f(slot, 1), a.dy_f + fidx, 4);
        cp_async(st.f(slot, 2), a.dz_f + fidx, 4);
        if (a.diffx) {
            cp_async(st.f(slot, 3), a.diffx + fidx, 4);
            cp_async(st.f(slot, 4), a.diffy + fidx, 4);
        }
        if (a.do_kodis) {
            cp_async(st.f(slot, 5), a.diffxx + fidx, 4);
            cp_async(st.f(slot, 6), a.diffyy + fidx, 4);
            cp_async(st.f(slot, 7), a.diffxy + fidx, 4);
        }
        if (a.do_bragg) {
            cp_async(st.ind(slot, 0), a.ind0_m + idx, 4);
            cp_async(st.ind(slot, 1), a.ind0_p + idx, 4);
        }
        if (load_scat) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < 2 * a.npol) cp_async(st.scat(slot, k), scat_buf + k * npix + idx, sizeof(T));
        }
    }
    // start the gathers of the scatterer-series values of the facet staged in `slot`
    template <typename A>
    static OCS_D void issue_gather(const A &a, const Stage<T> &st, int slot, int g) {
        int i0 = *st.ind(slot, 0) + a.tmod_m;
        i0 = i0 >= a.n_m ? i0 - a.n_m : i0;
        int i1 = *st.ind(slot, 1) + a.tmod_p;
        i1 = i1 >= a.n_p ? i1 - a.n_p : i1;
        if (sizeof(T) == 4 && a.s_m32) {
            cp_async(st.gather(g, 0), a.s_m32 + 2 * (long long)i0, 8);
            cp_async(st.gather(g, 1), a.s_p32 + 2 * (long long)i1, 8);
        } else {
            cp_async(st.gather(g, 0), a.s_m + 2 * (long long)i0, 16);
            cp_async(st.gather(g, 1), a.s_p + 2 * (long long)i1, 16);
        }
    }
    template <typename A>
    OCS_D void read(const A &a, const Stage<T> &st, int slot, bool load_scat) {
        dx = *st.f(slot, 0);
        dy = *st.f(slot, 1);
        dz = *st.f(slot, 2);
        if (a.diffx) { diffx = *st.f(slot, 3); diffy = *st.f(slot, 4); }
        if (a.do_kodis) { diffxx = *st.f(slot, 5); diffyy = *st.f(slot, 6); diffxy = *st.f(slot, 7); }
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            if (load_scat && p < a.npol) {
                scat[p][0] = *st.scat(slot, 2 * p);
                scat[p][1] = *st.scat(slot, 2 * p + 1);
            } else {
                scat[p][0] = (T)0;
                scat[p][1] = (T)0;
            }
        }
    }
};

template <typename T> OCS_D cplx<T> cexp_phase(double ph);
template <> OCS_D cplx<double> cexp_phase<double>(double ph) { return cexpi(ph); }
template <> OCS_D cplx<float> cexp_phase<float>(double ph) {
    float s, c;
    __sincosf((float)reduce_2pi(ph), &s, &c);
    return {c, s};
}

// Block-wide sum of a double; thread 0 adds it to *dst.
OCS_D void block_atomic_sum(double v, double *dst, double *sred) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sred[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += sred[i];
        if (s != 0.0) atomicAdd(dst, s);
    }
}

// Per-pulse row table (sar_raw_nompi.py:353-363, 485-493): for every facet row y,
// rowtab[q*ny + y] holds az, sin_az = az/sr0, the ground-projected azimuth angle and its
// cos / sin (q = 0..4), then rowtab[5*ny + 2*(y*nch + c)] the complex antenna-pattern x
// ATI-phase factor of channel c.  float64, computed once per pulse for all tiles.
OCS_D void pulse_row(const PulseArgs &a, double az_now, int y) {
    // the scatterometer's azimuth residual is float32 when the reference computes it from
    // a float32 grid step (numpy promotion), and then y - residual is a float32 difference
    const double az = a.az_f32 ? (double)__fsub_rn(a.y[y], (float)az_now) : dsub((double)a.y[y], az_now);
    const double sin_az = ddiv(az, a.sr0);
    const double azp = asin(az / a.gr0);
    a.rowtab[y] = az;
    a.rowtab[(long long)a.ny + y] = sin_az;
    a.rowtab[2LL * a.ny + y] = azp;
    a.rowtab[3LL * a.ny + y] = cos(azp);
    a.rowtab[4LL * a.ny + y] = sin(azp);
    const double bp = np_sinc(a.ltx_over_l * sin_az) * np_sinc(a.lrx_over_l * sin_az);
    double *fac = a.rowtab + 5LL * a.ny + 2LL * y * a.nch;
    for (int c = 0; c < a.nch; ++c) {
        const c128 ati = cexpi((-a.k0 * a.b_ati[c]) * sin_az);
        fac[2 * c] = bp * ati.re;
        fac[2 * c + 1] = bp * ati.im;
    }
}

// Shared memory of the pulse kernel: pre-shifted weight table, CTA bin window, the tile's
// rows of the per-pulse row table ([5][RCAP] float64 + [RCAP][nch] complex, RCAP = the
// largest tile height of the launch), and the block-reduction scratch.
template <typename T> struct PulseSmem {
    T *wtab, *bins;
    double *r_az;
    cplx<T> *r_fac;
    double *sred;
    Stage<T> stage;
};

template <typename T, int NOUT, int S, int RCAP>
OCS_HD constexpr size_t pulse_smem_bytes(int nch) {
    return (size_t)wtab_len<T, S>(kSincTaps, kSincOvs) * sizeof(T) + (size_t)NOUT * kPulseNbw * 2 * sizeof(T) +
           5 * RCAP * sizeof(double) + (size_t)RCAP * nch * sizeof(cplx<T>) + 32 * sizeof(double) +
           stage_bytes<T>();
}

template <typename T, int NOUT, int S, int RCAP>
OCS_D PulseSmem<T> pulse_smem(unsigned char *smem, int nch) {
    PulseSmem<T> sm;
    sm.wtab = reinterpret_cast<T *>(smem);
    sm.bins = sm.wtab + wtab_len<T, S>(kSincTaps, kSincOvs);             // [NOUT][nbw][2]
    sm.r_az = reinterpret_cast<double *>(sm.bins + NOUT * kPulseNbw * 2);
    sm.r_fac = reinterpret_cast<cplx<T> *>(sm.r_az + 5 * RCAP);            // [rows][nch]
    sm.sred = reinterpret_cast<double *>(sm.r_fac + RCAP * nch);
    const size_t st = reinterpret_cast<size_t>(sm.sred + 32);
    sm.stage.base = reinterpret_cast<unsigned char *>((st + 15) & ~(size_t)15);
    return sm;
}

// One tile of kPulseCols columns x tile_rows rows: NRCS, scene and accumulation of every
// facet into this pulse's raw rows; the tile's NRCS sums are added to spec_sum and
// bragg_sum.
template <typename T, int NOUT, int S, int RCAP, int MODE = kModeStd>
OCS_D void pulse_tile(const PulseArgs &a, int tile, int tile_rows, const PulseSmem<T> &sm, double &spec_sum,
                      double (&bragg_sum)[2]) {
    const int tiles_x = (a.nx + kPulseCols - 1) / kPulseCols;
    const int x = (tile % tiles_x) * kPulseCols + threadIdx.x;
    const int y0 = (tile / tiles_x) * tile_rows;
    const int nrows = min(tile_rows, a.ny - y0);
    __syncthreads();                    // previous tile's bins and row tables are consumed
    // this tile's rows of the per-pulse row table (pulse_rows_kernel)
    for (int i = threadIdx.x; i < nrows * 5; i += blockDim.x) {
        const int q = i / nrows, k = i - q * nrows;
        sm.r_az[q * RCAP + k] = a.rowtab[(long long)q * a.ny + y0 + k];
    }
    {
        const double *fac = a.rowtab + 5LL * a.ny + 2LL * y0 * a.nch;
        for (int i = threadIdx.x; i < nrows * a.nch; i += blockDim.x)
            sm.r_fac[i] = {(T)fac[2 * i], (T)fac[2 * i + 1]};
    }

    CtaBins<T, NOUT> cb;
    cb.acc = sm.bins;
    cb.nbw = kPulseNbw;
    cb.nout = a.nout;
    cb.nbins = a.nbins;
    cb.out = reinterpret_cast<T *>(a.raw) + 2 * ((long long)a.out0 * a.raw_out_stride + a.raw_row);
    if constexpr ((MODE & kModeSkim) != 0) cb.out += 2 * (long long)(y0 / a.ny_integ) * a.nbins;
    cb.out_stride = a.raw_out_stride;
    {
        // window base: bin of this CTA's first column at its first row, undisplaced
        const int xc = min((tile % tiles_x) * kPulseCols, a.nx - 1);
        const double az = (double)a.y[y0] - a.az_now;
        const double srg = a.sr_col[xc] + az * 0.5 * (az / a.sr0) + a.sr_bin_off;
        cb.cta_base = (int)floor((srg - a.min_sr) / a.binsize) - 24;
    }
    cb.zero();
    __syncthreads();

    BinWindow<T, S, NOUT> win;
    win.reset();
    if (x < a.nx) {
        const double sr_c = a.sr_col[x], sin_i = a.sin_inc[x], cos_i = a.cos_inc[x];
        const double inc_c = a.inc[x];
        const double dinc0 = inc_c - a.inc_angle;
        const double tan_i = a.do_kodis ? a.tan_inc[x] : 0.0;
        double cap = 0.0;
        if (a.do_bragg) {
            if constexpr ((MODE & kModeSca)) cap = dmul(dmul(2.0 * a.k0, a.c_b[x]), a.cap_t);
            else cap = ((2.0 * a.k0) * a.t_step) * a.c_b[x] * (double)(a.az_step + 1);
        }
        const float cap_r = (float)reduce_2pi(cap);
        const double two_k0 = 2.0 * a.k0;
        const long long npix = (long long)a.nx * a.ny;
        T *scat = reinterpret_cast<T *>(a.scat);
        const bool load_scat = a.do_bragg && !(MODE & kModeSca);
        // software pipeline through shared memory: the inputs of the next rows and
        // the scatterer-series gathers of row i + 1 are in flight while row i is processed
        const Stage<T> &st = sm.stage;
        const long long idx0 = (long long)y0 * a.nx + x;
        // outputs of this pass, 5 bits each: channel (bits 0-2), polarisation (bit 3) and
        // whether the channel has an XTI phase (bit 4)
        unsigned outs = 0;
#pragma unroll
        for (int k = 0; k < NOUT; ++k) {
            const int o = a.out0 + k;
            const int p = o / a.nch, c = o - p * a.nch;
            const bool xti = k < a.nout && a.b_xti[c] != 0.0;
            outs |= (unsigned)(c | (p << 3) | (xti ? 16 : 0)) << (5 * k);
        }
        // indices of tile row r: per-facet arrays (ridx) and surface fields (fidx); the
        // scatterometer mode reads the fields of the rolled row and the column mod fnx
        int fx = x;
        if constexpr ((MODE & kModeSca)) fx = x % a.fnx;
        auto row_index = [&](int r, long long &ridx, long long &fidx) {
            if constexpr ((MODE & kModeSca)) {
                int fr = y0 + r + a.roll;
                fr = fr >= a.ny ? fr - a.ny : fr;
                ridx = (long long)fr * a.nx + x;
                fidx = (long long)fr * a.fnx + fx;
            } else {
                ridx = idx0 + (long long)r * a.nx;
                fidx = ridx;
            }
        };
        auto issue_row = [&](int r, int slot) {
            if (r < nrows) {
                long long ridx, fidx;
                row_index(r, ridx, fidx);
                FacetIn<T>::issue(a, st, slot, ridx, npix, scat, load_scat, fidx);
            }
            cp_async_commit();
        };
        FacetIn<T> cur;
        if constexpr (stage_rows<T>() == 4) {
            // Commit order: rows 0, 1; gathers of row 0; row 2; then per row i the gathers of
            // row i + 1 and row i + 3.  Waiting for all groups but the newest at the top of
            // row i completes rows <= i + 1 and the gathers of row i and leaves row i + 2 in
            // flight, so two rows of inputs are on their way while a row is processed.
            issue_row(0, 0);
            issue_row(1, 1);
            cp_async_wait<1>();
            if (a.do_bragg) FacetIn<T>::issue_gather(a, st, 0, 0);
            cp_async_commit();
            issue_row(2, 2);
        } else {
            // rows 0, 1, then gathers of row 0; per row i: row i + 2, gathers of row i + 1
            issue_row(0, 0);
            issue_row(1, 1);
            cp_async_wait<1>();
            if (a.do_bragg) FacetIn<T>::issue_gather(a, st, 0, 0);
            cp_async_commit();
        }
        int slot_i = 0;
        for (int i = 0; i < nrows; ++i) {
            int slot_n;
            if constexpr (stage_rows<T>() == 4) {
                slot_n = (i + 1) & 3;
                cp_async_wait<1>();             // rows <= i + 1 and the gathers of row i have landed
                if (a.do_bragg && i + 1 < nrows) FacetIn<T>::issue_gather(a, st, slot_n, (i + 1) & 1);
                cp_async_commit();
                issue_row(i + 3, (i + 3) & 3);  // into the slot of row i - 1
            } else {
                slot_n = slot_i == 2 ? 0 : slot_i + 1;
                issue_row(i + 2, slot_i == 0 ? 2 : slot_i - 1);
                cp_async_wait<1>();             // rows <= i + 1 and the gathers of row i have landed
                if (a.do_bragg && i + 1 < nrows) FacetIn<T>::issue_gather(a, st, slot_n, (i + 1) & 1);
                cp_async_commit();
            }
            cur.read(a, st, slot_i, load_scat);
            slot_i = slot_n;
            // SKIM calibration target: a fixed one sits at zero displacement (skim_raw.py:490-493)
            const bool pt_here = (MODE & kModeSkim) && a.pt_mode != 0 && y0 + i == a.pt_y && x == a.pt_x;
            if (pt_here && a.pt_mode == 2) {
                cur.dx = 0.f;
                cur.dy = 0.f;
                cur.dz = 0.f;
            }
            const double az = sm.r_az[i];
            // SKIM: sin_az = az / sr of this facet's column (skim_raw.py:486)
            const double sin_az = (MODE & kModeSkim) ? ddiv(az, sr_c) : sm.r_az[RCAP + i];
            // slant range: sr - cos_inc*Dz + az/2*sin_az + Dx*sin_inc + Dy*sin_az, float64,
            // left to right, no fused multiply-adds (bit-identical with numpy); the SKIM
            // two-scale form leaves az/2*sin_az out of the phase range (skim_raw.py:494-505)
            double srs = dsub(sr_c, dmul(cos_i, (double)cur.dz));
            if (!(MODE & kModeSkim) || a.skim_az2) srs = dadd(srs, dmul(az * 0.5, sin_az));
            srs = dadd(srs, dmul((double)cur.dx, sin_i));
            srs = dadd(srs, dmul((double)cur.dy, sin_az));
            int bin_d, lut;
            {
                // the scatterometer's sub-pulses arrive later by sr_bin_off; the SKIM
                // two-scale form with rcm adds az/2*sin_az to the bins only
                double srb = ((MODE & kModeSca)) ? dadd(srs, a.sr_bin_off) : srs;
                if ((MODE & kModeSkim) && a.skim_rcm) srb = dadd(srs, dmul(az * 0.5, sin_az));
                if (sizeof(T) == 8) bin_and_lut(srb, a.min_sr, a.binsize, kSincOvs, bin_d, lut);
                else bin_and_lut_fast(srb, a.min_sr, a.inv_binsize, kSincOvs, bin_d, lut);
            }
            // two-way spreading of the scatterometer scene, (sr0 / (sr0 + r))^2
            T rscale = (T)1;
            if constexpr ((MODE & kModeSca)) {
                const double q = ddiv(a.sr0, dadd(a.sr0, srs));
                rscale = (T)dmul(q, q);
            }

            cplx<T> scene[2] = {{(T)0, (T)0}, {(T)0, (T)0}};      // per polarisation
            if constexpr ((MODE & kModeKa) != 0) {
                c128 last = {0.0, 0.0};
                for (int p = 0; p < a.npol; ++p) {
                    const int pc = a.rom.pol == POL_DP ? p : (a.rom.pol == POL_HH ? 0 : 1);
                    last = ka_specular(a.ka, pc, srs, (double)a.x_f[fx], (double)a.y[y0 + i], sin_i, cos_i, tan_i,
                                       sm.r_az[4 * RCAP + i], sm.r_az[3 * RCAP + i], cur.dz, cur.diffx, cur.diffy,
                                       cur.diffxx, cur.diffyy, cur.diffxy);
                    scene[p] = {(T)last.re, (T)last.im};
                    // the scatterometer scales the field by the two-way spreading
                    if constexpr ((MODE & kModeSca) != 0) scene[p] = {scene[p].re * rscale, scene[p].im * rscale};
                }
                spec_sum += last.re * last.re + last.im * last.im;
            } else if (a.do_kodis) {
                const cplx<T> e = kodis_facet<T>(a.kodis, srs, sin_i, cos_i, tan_i, sm.r_az[3 * RCAP + i], sm.r_az[4 * RCAP + i],
                                                 cur.diffx, cur.diffy, cur.diffxx, cur.diffyy, cur.diffxy);
                const T s4 = (T)3.5449077018110318;                 // sqrt(4 pi)
                const cplx<T> es = {e.re * s4, e.im * s4};
                spec_sum += (double)es.re * es.re + (double)es.im * es.im;
                if constexpr ((MODE & kModeSca)) {
                    scene[0] = {es.re * rscale, es.im * rscale};
                    scene[1] = scene[0];
                } else {
                    scene[0] = es;
                    scene[1] = es;
                }
            }
            if (a.do_bragg) {
                T sc[2][2];                                            // [pol][line]
                if constexpr ((MODE & kModeSca) != 0) {
                    // the scatterometer evaluates the model on every launch and stores nothing
                    T hh[2], vv[2];
                    if (a.lut) {
                        // the table holds the model's output polarisation(s) in output order
                        const int ai = lut_az_index(a, sm.r_az[2 * RCAP + i]);
                        // the scatterometer's range blocks each have their own table
                        const long long tb = (long long)(x / a.fnx) * a.lut_block;
                        T r0[2], r1[2];
                        romeiser_lut<T>(a, ai, cur.diffx, cur.diffy, 0, r0, tb);
                        if (a.npol == 2) romeiser_lut<T>(a, ai, cur.diffx, cur.diffy, 1, r1, tb);
                        else { r1[0] = r0[0]; r1[1] = r0[1]; }
                        const bool vv_first = a.rom.pol == POL_VV;
                        hh[0] = vv_first ? r1[0] : r0[0]; hh[1] = vv_first ? r1[1] : r0[1];
                        vv[0] = vv_first ? r0[0] : r1[0]; vv[1] = vv_first ? r0[1] : r1[1];
                    } else {
                        romeiser_facet<T>(a.rom, (T)inc_c, (T)sm.r_az[2 * RCAP + i], (T)sm.r_az[3 * RCAP + i],
                                          (T)sm.r_az[4 * RCAP + i], (T)cur.diffx, (T)cur.diffy, hh, vv);
                    }
                    if (a.use_hmtf) {
                        // weighted by 1 + hMTF of the rolled row, unclipped (the reference's clipping
                        // writes land in the unrolled surface, dopsca_raw.py:463-472)
                        long long ridx_h, fidx_h;
                        row_index(i, ridx_h, fidx_h);
                        const float hm = a.hmtf[fidx_h];
                        const T f = (T)(1.f + hm);
                        hh[0] *= f; hh[1] *= f; vv[0] *= f; vv[1] *= f;
                    }
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        if (p < a.npol) {
                            const bool use_vv = a.rom.pol == POL_VV || (a.rom.pol == POL_DP && p == 1);
                            const T r0 = use_vv ? vv[0] : hh[0], r1 = use_vv ? vv[1] : hh[1];
                            bragg_sum[p] += (double)r0 + (double)r1;
                            sc[p][0] = tsqrt(r0);
                            sc[p][1] = tsqrt(r1);
                        }
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < 2; ++p) { sc[p][0] = cur.scat[p][0]; sc[p][1] = cur.scat[p][1]; }
                }
                // Bragg phases: -2 k0 r -/+ 2 k0 t_step c_b (az_step + 1)
                cplx<T> e0, e1;
                if (sizeof(T) == 8) {
                    const double surf = (-two_k0) * srs;
                    e0 = cexp_phase<T>(surf - cap);
                    e1 = cexp_phase<T>(surf + cap);
                } else {
                    const float rs = (float)reduce_2pi((-two_k0) * srs);
                    float s0, c0, s1, c1;
                    __sincosf(rs - cap_r, &s0, &c0);
                    __sincosf(rs + cap_r, &s1, &c1);
                    e0 = {(T)c0, (T)s0};
                    e1 = {(T)c1, (T)s1};
                }
                cplx<T> sm, sp;
                if (sizeof(T) == 4 && a.s_m32) {
                    const float2 smf = *reinterpret_cast<const float2 *>(st.gather(i & 1, 0));
                    const float2 spf = *reinterpret_cast<const float2 *>(st.gather(i & 1, 1));
                    sm = {(T)smf.x, (T)smf.y};
                    sp = {(T)spf.x, (T)spf.y};
                } else {
                    const double2 smd = *st.gather(i & 1, 0);
                    const double2 spd = *st.gather(i & 1, 1);
                    sm = {(T)smd.x, (T)smd.y};
                    sp = {(T)spd.x, (T)spd.y};
                }
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    if (p < a.npol) {
                        const cplx<T> l0 = cmul(cplx<T>{sc[p][0] * e0.re, sc[p][0] * e0.im}, sm);
                        const cplx<T> l1 = cmul(cplx<T>{sc[p][1] * e1.re, sc[p][1] * e1.im}, sp);
                        cplx<T> lb = cadd(l0, l1);
                        if constexpr ((MODE & kModeSca)) lb = {lb.re * rscale, lb.im * rscale};
                        scene[p] = cadd(scene[p], lb);
                    }
                }
            }
            if (pt_here) {
                // the target replaces the facet's scene value: pt_amp exp(-2 i k0 r)
                // (skim_raw.py:608-615), float64 like the reference's complex128 scene
                double ps, pc;
                sincos((-two_k0) * srs, &ps, &pc);
                for (int p = 0; p < a.npol; ++p) scene[p] = {(T)(a.pt_amp * pc), (T)(a.pt_amp * ps)};
            }
            // channels of this pass: antenna pattern x ATI phase (per row) x XTI phase
            cplx<T> coef[NOUT];
            double wave_dinc = 0.0;
            if (a.any_xti) wave_dinc = ((double)cur.dz * sin_i + (double)cur.dx * sin_i) / a.sr0;
            T bp_f = (T)1;
            if constexpr ((MODE & kModeSkim) != 0) {
                // two-way antenna pattern of this facet, power units for both the transmit
                // and the receive pattern (antenna.py:28-42 passes its field flag to the
                // positional catch-all of sinc_bp)
                T tx, rx;
                if constexpr (sizeof(T) == 8) {
                    tx = np_sinc(a.atx * sin_az);
                    rx = np_sinc(a.arx * sin_az);
                } else {
                    tx = np_sinc((float)(a.atx * sin_az));
                    rx = np_sinc((float)(a.arx * sin_az));
                }
                bp_f = (tx * tx) * (rx * rx);
            }
#pragma unroll
            for (int k = 0; k < NOUT; ++k) {
                if (k < a.nout) {
                    const unsigned ok = outs >> (5 * k);
                    const int c = ok & 7;
                    cplx<T> v;
                    if constexpr ((MODE & kModeSkim) != 0) {
                        const cplx<T> sc = (ok & 8) ? scene[1] : scene[0];
                        v = {sc.re * bp_f, sc.im * bp_f};
                    } else {
                        v = cmul((ok & 8) ? scene[1] : scene[0], sm.r_fac[i * a.nch + c]);
                    }
                    if (ok & 16) {
                        const double ph = (-a.k0 * a.b_xti[c]) * (dinc0 + wave_dinc);
                        v = cmul(v, cexp_phase<T>(ph));
                    }
                    coef[k] = v;
                } else {
                    coef[k] = {(T)0, (T)0};
                }
            }
            if (bin_d > -(1 << 29))
                win.add(bin_d - mode_taps<MODE>() / 2, lut, coef, sm.wtab, a.sinc, mode_taps<MODE>(), kSincOvs, cb);
        }
        cp_async_wait<0>();
    }
    if constexpr ((MODE & kModeSca)) {
        // the scatterometer's NRCS sums are kept per range block: each column adds its
        // tile's sums to its block
        if (x < a.nx) {
            const long long blk = x / a.fnx;
            if (a.do_kodis && spec_sum != 0.0) atomicAdd(&a.nrcs_spec[(long long)a.nrcs_row * a.nblk + blk], spec_sum);
            if (a.do_bragg)
                for (int p = 0; p < a.npol; ++p)
                    if (bragg_sum[p] != 0.0)
                        atomicAdd(&a.nrcs_bragg[((long long)p * a.nrcs_rows + a.nrcs_row) * a.nblk + blk], bragg_sum[p]);
        }
        spec_sum = 0.0;
        bragg_sum[0] = bragg_sum[1] = 0.0;
    }
    win.flush(cb);
    __syncthreads();
    cb.flush_to_global();
}

// NRCS bookkeeping of a CTA (only the first output group accumulates it).
template <typename T>
OCS_D void pulse_nrcs(const PulseArgs &a, const PulseSmem<T> &sm, double spec_sum) {
    if (a.out0 == 0) {
        if (a.do_kodis) block_atomic_sum(spec_sum, &a.nrcs_spec[a.az_step], sm.sred);
    }
}

template <typename T, int NOUT, int S, int MODE>
__global__ void __launch_bounds__(kPulseCols, (sizeof(T) == 4 && NOUT < 4) ? 4 : 2)
pulse_kernel(const __grid_constant__ PulseArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const PulseSmem<T> sm = pulse_smem<T, NOUT, S, kPulseRows>(smem, a.nch);
    build_wtab<T, S>(sm.wtab, a.sinc, mode_taps<MODE>(), kSincOvs);
    const int tiles = ((a.nx + kPulseCols - 1) / kPulseCols) * ((a.ny + a.tile_rows - 1) / a.tile_rows);
    double spec_sum = 0.0, bragg_sum[2] = {0.0, 0.0};
    // persistent CTAs: each walks tiles of kPulseCols columns x tile_rows rows
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x)
        pulse_tile<T, NOUT, S, kPulseRows, MODE>(a, tile, a.tile_rows, sm, spec_sum, bragg_sum);
    pulse_nrcs<T>(a, sm, spec_sum);
}

// ---------------------------------------------------------------------------------------
// Scene batch (batch.cuh).  Output groups: a slot's npol*nch outputs are taken G at a time
// (G = 4 in the mixed form, 2 in FP64); a group of w outputs runs in the kernel of width
// class 1 (w = 1), 2 (w = 2) or 4 (w = 3, 4).  The step's refresh items have stored sqrt(RCS)
// before any group reads it.
OCS_HD constexpr int width_class(int w) { return w <= 1 ? 1 : (w == 2 ? 2 : 4); }

// Number of groups of width class K among nout outputs; out0 / width of the j-th one.
OCS_D int groups_of_class(int nout, int G, int K, int j, int &out0, int &width) {
    int n = 0;
    for (int o = 0; o < nout; o += G) {
        const int w = nout - o < G ? nout - o : G;
        if (width_class(w) == K) {
            if (n == j) { out0 = o; width = w; }
            ++n;
        }
    }
    return n;
}

OCS_D int slot_pulse_tiles(const SlotState &g) {
    return ((g.nx + kPulseCols - 1) / kPulseCols) * ((g.ny + g.tile_rows - 1) / g.tile_rows);
}

// Row quantities of a tile, evaluated by the CTA itself (the fine-grid kernels): the values of
// pulse_row for the rows y0 .. y0 + nrows - 1 and the outputs of the pass, split into
// independent tasks (azimuth angle; the two antenna patterns; one ATI phase per output) so
// that their float64 chains run side by side.  A separate row-table launch cost 3 us per pulse
// (float64) to 6 us (mixed), a fifth to a third of a pulse on small surfaces.
//   tmp (shared): [nrows][2 + 2 nout] patterns and ATI factors;
//   row(r, az, sin_az, azp, cos_azp, sin_azp) is called once per row by one thread;
// after a barrier, tile_factor(tmp, ...) gives an output's complex factor of a row.
template <int NOUT, class Row>
OCS_D void eval_tile_rows(const PulseArgs &a, int y0, int nrows, double *tmp, const Row &row) {
    constexpr int W = 2 + 2 * NOUT;
    const int tasks = 3 + a.nout;
    for (int i = threadIdx.x; i < nrows * tasks; i += blockDim.x) {
        const int q = i / nrows, r = i - q * nrows;           // lanes share a task
        const double az = dsub((double)a.y[y0 + r], a.az_now);
        const double sin_az = ddiv(az, a.sr0);
        if (q == 0) {
            const double azp = asin(az / a.gr0);
            row(r, az, sin_az, azp, cos(azp), sin(azp));
        } else if (q < 3) {
            tmp[r * W + q - 1] = np_sinc((q == 1 ? a.ltx_over_l : a.lrx_over_l) * sin_az);
        } else {
            const int k = q - 3, c = (a.out0 + k) % a.nch;
            const c128 ati = cexpi((-a.k0 * a.b_ati[c]) * sin_az);
            tmp[r * W + 2 + 2 * k] = ati.re;
            tmp[r * W + 3 + 2 * k] = ati.im;
        }
    }
}
template <int NOUT> OCS_D c128 tile_factor(const double *tmp, int r, int k) {
    const double *t = tmp + r * (2 + 2 * NOUT);
    const double bp = t[0] * t[1];
    return {bp * t[2 + 2 * k], bp * t[3 + 2 * k]};
}

// Range bins that the 128 columns of a tile span on a flat sea.
inline double tile_span(double facet_dx, double inc_angle, double binsize) {
    return kPulseCols * facet_dx * fabs(sin(inc_angle)) / binsize;
}
// Whether the fine grid holds a tile's bins: the span has to leave a quarter of it for the azimuth
// curvature of the rows and the waves' displacements.
inline bool grid_holds_tile(double span) { return span <= 0.75 * kGridBins; }

// Tile height for a persistent launch: the tallest (<= kPulseRows) that still gives every
// resident CTA slot a tile in the last wave, at least `least` rows.
inline int tile_rows_for(int nx, int ny, int cols, int resident, int least) {
    const int tiles_x = (nx + cols - 1) / cols;
    const long long want = (long long)resident * (((long long)tiles_x * ((ny + kPulseRows - 1) / kPulseRows) +
                                                   resident - 1) / resident);
    long long per_col = want / tiles_x;
    if (per_col < 1) per_col = 1;
    const int rows = (int)((ny + per_col - 1) / per_col);
    return rows < least ? (ny < least ? ny : least) : (rows > kPulseRows ? kPulseRows : rows);
}

// Launches of pulse_general.cu: the output group [a.out0, a.out0 + a.nout) of one pulse, and one
// batch class, on the float64-range kernel.
int launch_pulse_general(const PulseArgs &a, int precision, cudaStream_t st);
int batch_pulse_general(const BatchRef &b, int precision, int kind, int width, int grid, cudaStream_t st);

}  // namespace ocs
