// Entry points of one radar pulse (pulse_core.cuh, pulse_mixed.cuh): descriptor checks, per-
// pulse row tables, tensor maps and the dispatch to the launches of pulse_general.cu and
// pulse_split.cu.
#include <cudaTypedefs.h>
#include <string.h>

#include <mutex>

#include "pulse_f64.cuh"
#include "pulse_mixed.cuh"
#include "pulse_refresh.cuh"

namespace ocs {

__global__ void pulse_rows_kernel(const __grid_constant__ PulseArgs a) {
    for (int y = blockIdx.x * blockDim.x + threadIdx.x; y < a.ny; y += gridDim.x * blockDim.x)
        pulse_row(a, a.az_now, y);
}

__global__ void pulse_rows_mixed_kernel(const __grid_constant__ PulseArgs a, float *lo_row, int nout_all) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned char *ws = reinterpret_cast<unsigned char *>(a.rowtab);
    int *hdr = reinterpret_cast<int *>(ws + mix_hdr_offset(a.ny, a.nch));
    if (t < a.ny) mix_row(a, a.az_now, t);
    // fold the compensation row of the previous pulse (pending >= 0) into its raw row
    if (lo_row) {
        const int pending = hdr[0];
        const long long nfold = (long long)nout_all * a.nbins;
        if (pending >= 0) {
            float *raw = reinterpret_cast<float *>(a.raw);
            for (long long i = t; i < nfold; i += (long long)gridDim.x * blockDim.x) {
                const long long o = i / a.nbins, b = i - o * a.nbins;
                float *dst = raw + 2 * (o * a.raw_out_stride + (long long)pending * a.nbins + b);
                const float lr = lo_row[2 * i], li = lo_row[2 * i + 1];
                if (lr != 0.f) dst[0] += lr;
                if (li != 0.f) dst[1] += li;
                lo_row[2 * i] = 0.f;
                lo_row[2 * i + 1] = 0.f;
            }
        }
    }
}

// The fold alone (end of a scene, or before the raw cube is read).
__global__ void pulse_flush_kernel(const __grid_constant__ PulseArgs a, float *lo_row, int nout_all) {
    grid_wait();
    unsigned char *ws = reinterpret_cast<unsigned char *>(a.rowtab);
    int *hdr = reinterpret_cast<int *>(ws + mix_hdr_offset(a.ny, a.nch));
    const int pending = hdr[0];
    const long long nfold = (long long)nout_all * a.nbins;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (pending >= 0) {
        float *raw = reinterpret_cast<float *>(a.raw);
        for (long long i = t; i < nfold; i += (long long)gridDim.x * blockDim.x) {
            const long long o = i / a.nbins, b = i - o * a.nbins;
            float *dst = raw + 2 * (o * a.raw_out_stride + (long long)pending * a.nbins + b);
            const float lr = lo_row[2 * i], li = lo_row[2 * i + 1];
            if (lr != 0.f) dst[0] += lr;
            if (li != 0.f) dst[1] += li;
            lo_row[2 * i] = 0.f;
            lo_row[2 * i + 1] = 0.f;
        }
    }
}

// Tensor-map encoder of the driver, resolved once through the runtime (no link to libcuda).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// One map of a [depth][ny][nx] tensor of 4-byte elements with planes `plane` bytes apart
// and boxes of one row of kMixCols columns times `depth` planes (depth 1: two-dimensional).
static bool encode_rows_map(CUtensorMap &m, const void *base, CUtensorMapDataType type, int nx, int ny, int depth,
                            unsigned long long plane) {
    PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc) return false;
    const cuuint32_t rank = depth > 1 ? 3 : 2;
    const cuuint64_t dims[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)depth};
    const cuuint64_t strides[2] = {(cuuint64_t)nx * 4, (cuuint64_t)plane};
    const cuuint32_t box[3] = {(cuuint32_t)kMixCols, 1, (cuuint32_t)depth};
    const cuuint32_t estr[3] = {1, 1, 1};
    return enc(&m, type, rank, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Whether a pulse's inputs suit the split-range kernel: fields equally spaced in one
// allocation, 16-byte aligned bases and nx a multiple of 4 (every row of every input then
// starts on a 16-byte boundary, as its tensor copies and 8-byte loads need).
static bool mix_inputs_ok(const ocs_pulse_desc *d) {
    if (d->nx % 4 != 0 || d->nx < 4) return false;
    const int nf = d->do_kodis ? 8 : 5;
    const char *f[8] = {(const char *)d->dx_d, (const char *)d->dy_d, (const char *)d->dz_d,
                        (const char *)d->diffx_d, (const char *)d->diffy_d, (const char *)d->diffxx_d,
                        (const char *)d->diffyy_d, (const char *)d->diffxy_d};
    const long long plane = (long long)(f[1] - f[0]);
    const long long need = (long long)d->nx * d->ny * 4;
    if (plane < need || plane % 16 != 0 || ((uintptr_t)f[0] & 15)) return false;
    for (int k = 1; k < nf; ++k)
        if (!f[k] || f[k] - f[0] != k * plane) return false;
    return !d->do_bragg || !((((uintptr_t)d->ind0_m_d) | ((uintptr_t)d->ind0_p_d) | ((uintptr_t)d->scat_d)) & 15);
}

// Tensor maps of a pulse descriptor that passed mix_inputs_ok (register-window form).
static bool fill_mix_maps(const ocs_pulse_desc *d, MixMaps &m) {
    memset(&m, 0, sizeof(m));
    m.nf = d->do_kodis ? 8 : 5;
    const unsigned long long plane = (unsigned long long)((const char *)d->dy_d - (const char *)d->dx_d);
    if (!encode_rows_map(m.fields, d->dx_d, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, d->nx, d->ny, m.nf, plane)) return false;
    if (!d->do_bragg) return true;
    return encode_rows_map(m.indm, d->ind0_m_d, CU_TENSOR_MAP_DATA_TYPE_INT32, d->nx, d->ny, 1, 0) &&
           encode_rows_map(m.indp, d->ind0_p_d, CU_TENSOR_MAP_DATA_TYPE_INT32, d->nx, d->ny, 1, 0) &&
           encode_rows_map(m.scat, d->scat_d, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, d->nx, d->ny, 2 * d->npol,
                           (unsigned long long)d->nx * d->ny * 4);
}

}  // namespace ocs

using namespace ocs;

static int fill_pulse_args(const ocs_pulse_desc *d, PulseArgs &a) {
    memset(&a, 0, sizeof(a));
    if (!d || d->nx < 1 || d->ny < 1 || d->npol < 1 || d->npol > 2 || d->nch < 1 || d->nch > kMaxCh)
        return OCS_ERR_ARG;
    if (!d->dx_d || !d->dy_d || !d->dz_d || !d->y_d || !d->sr_col_d || !d->sin_inc_d || !d->cos_inc_d ||
        !d->inc_d || !d->sinc_d || !d->raw_d)
        return OCS_ERR_ARG;
    if (d->do_kodis && (!d->diffx_d || !d->diffy_d || !d->diffxx_d || !d->diffyy_d || !d->diffxy_d ||
                        !d->tan_inc_d || !d->nrcs_spec_d))
        return OCS_ERR_ARG;
    if (d->do_bragg && (!d->diffx_d || !d->diffy_d || !d->c_b_d || (!d->scat_d && !d->sca) || !d->s_m_d || !d->s_p_d ||
                        !d->ind0_m_d || !d->ind0_p_d || d->n_m < 1 || d->n_p < 1 || !d->spec_k_d ||
                        !d->spec_s_d || d->spec_n < 2 || !d->nrcs_bragg_d))
        return OCS_ERR_ARG;
    if (d->do_bragg && d->use_hmtf && !d->hmtf_d) return OCS_ERR_ARG;
    if (d->az_step < 0 || d->az_step >= d->az_steps || d->nbins < 1 || !d->rowtab_d) return OCS_ERR_ARG;
    if ((d->npol == 2) != (d->pol == POL_DP)) return OCS_ERR_ARG;
    a.nx = d->nx; a.ny = d->ny; a.npol = d->npol; a.nch = d->nch;
    a.dx_f = d->dx_d; a.dy_f = d->dy_d; a.dz_f = d->dz_d;
    a.diffx = d->diffx_d; a.diffy = d->diffy_d;
    a.diffxx = d->diffxx_d; a.diffyy = d->diffyy_d; a.diffxy = d->diffxy_d; a.hmtf = d->hmtf_d;
    a.y = d->y_d;
    a.sr_col = d->sr_col_d; a.sin_inc = d->sin_inc_d; a.cos_inc = d->cos_inc_d; a.tan_inc = d->tan_inc_d;
    a.inc = d->inc_d; a.c_b = d->c_b_d;
    a.inc_angle = d->inc_angle; a.sr0 = d->sr0; a.gr0 = d->gr0; a.k0 = d->k0; a.az_now = d->az_now;
    a.min_sr = d->min_sr; a.binsize = d->binsize; a.inv_binsize = 1.0 / d->binsize;
    a.t_step = d->t_step; a.az_step = d->az_step;
    a.tind = d->tind;
    a.ltx_over_l = d->ant_l_tx * d->f0 / 2.99792458e8;
    a.lrx_over_l = d->ant_l_rx * d->f0 / 2.99792458e8;
    for (int c = 0; c < d->nch; ++c) {
        a.b_ati[c] = d->b_ati[c];
        a.b_xti[c] = d->b_xti[c];
        if (d->b_xti[c] != 0.0) a.any_xti = 1;
    }
    a.do_kodis = d->do_kodis; a.do_bragg = d->do_bragg; a.refresh = d->refresh; a.use_hmtf = d->use_hmtf;
    a.kodis.k0 = d->k0;
    a.kodis.R_re = d->kodis_R_re; a.kodis.R_im = d->kodis_R_im;
    a.kodis.hdx = (double)d->facet_dx * 0.5; a.kodis.hdy = (double)d->facet_dy * 0.5;
    a.f_inv_bs = (float)a.inv_binsize;
    a.f_khi = (float)(2.0 * a.k0);
    a.f_klo = (float)(2.0 * a.k0 - (double)a.f_khi);
    a.f_hdx = (float)a.kodis.hdx; a.f_hdy = (float)a.kodis.hdy;
    a.f_inv_sr0 = (float)(1.0 / a.sr0);
    a.f_hr = (float)(0.5 * a.kodis.R_re); a.f_hi = (float)(0.5 * a.kodis.R_im);
    for (int c = 0; c < d->nch; ++c) a.f_kxti[c] = (float)(-a.k0 * a.b_xti[c]);
    RomeiserParams &r = a.rom;
    r.k0 = d->k0; r.d = d->bragg_d; r.dx = (double)d->facet_dx; r.dy = (double)d->facet_dy;
    r.wind_dir = d->wind_dir; r.wind_U = d->wind_U; r.pol = d->pol; r.spread = d->spread;
    r.ck_p = d->spread_ck_p; r.ck_m = d->spread_ck_m; r.a0 = d->spread_a0; r.ap = d->spread_ap;
    r.am = d->spread_am;
    r.tab_k = d->spec_k_d; r.tab_s = d->spec_s_d; r.tab_n = d->spec_n;
    r.eps_re = 73.0; r.eps_im = 18.0;
    r.seps_re = d->sqrt_eps_re; r.seps_im = d->sqrt_eps_im;
    r.eps2_re = 73.0 * 73.0 - 18.0 * 18.0; r.eps2_im = 2.0 * 73.0 * 18.0;
    a.scat = d->scat_d; a.s_m = d->s_m_d; a.s_p = d->s_p_d;
    if (d->s_m32_d && d->s_p32_d) { a.s_m32 = d->s_m32_d; a.s_p32 = d->s_p32_d; }
    if (d->do_bragg) {
        if (d->n_m > (1LL << 30) || d->n_p > (1LL << 30) || d->tind < 0) return OCS_ERR_SIZE;
        a.n_m = (int)d->n_m; a.n_p = (int)d->n_p;
        a.tmod_m = (int)(d->tind % d->n_m); a.tmod_p = (int)(d->tind % d->n_p);
    }
    a.ind0_m = d->ind0_m_d; a.ind0_p = d->ind0_p_d;
    a.sinc = d->sinc_d;
    a.raw = d->raw_d;
    a.rowtab = (double *)d->rowtab_d;
    a.nbins = d->nbins;
    a.raw_out_stride = (long long)d->az_steps * d->nbins;
    a.raw_row = (long long)d->az_step * d->nbins;
    a.nrcs_spec = d->nrcs_spec_d; a.nrcs_bragg = d->nrcs_bragg_d; a.az_steps = d->az_steps;
    a.spec_mode = d->do_kodis ? d->spec_mode : 0;
    if (a.spec_mode < 0 || a.spec_mode > 2) return OCS_ERR_ARG;
    if (a.spec_mode != 0 && !d->x_d) return OCS_ERR_ARG;
    a.x_f = d->x_d;
    a.ka.k0 = d->k0; a.ka.dx = d->ka_dx; a.ka.dy = d->ka_dy; a.ka.K_re = d->ka_K_re; a.ka.K_im = d->ka_K_im;
    a.ka.mode = a.spec_mode == 2 ? 1 : 0;
    if (d->skim) {
        // SKIM mode: one channel; the facets of every skim_ny_integ rows go to their
        // own output row: raw_d holds [npol][az_steps][ny / skim_ny_integ][nbins]
        if (d->sca || d->nch != 1 || d->skim_ny_integ < 1 || d->ny % d->skim_ny_integ != 0) return OCS_ERR_ARG;
        if (d->skim_ny_integ > kPulseRows && d->skim_ny_integ < d->ny) {
            for (int n = d->skim_ny_integ; n > kPulseRows; n /= 2)
                if (n % 2) return OCS_ERR_ARG;
        }
        a.skim = 1;
        a.ny_integ = d->skim_ny_integ;
        a.s_int = d->ny / d->skim_ny_integ;
        a.skim_az2 = d->skim_az2 != 0;
        a.skim_rcm = d->skim_rcm != 0;
        if (d->pt_mode < 0 || d->pt_mode > 2) return OCS_ERR_ARG;
        a.pt_mode = d->pt_mode;
        a.pt_x = d->pt_x;
        a.pt_y = d->pt_y;
        a.pt_amp = d->pt_amp;
        a.atx = a.ltx_over_l;
        a.arx = a.lrx_over_l;
        a.raw_out_stride = (long long)d->az_steps * a.s_int * d->nbins;
        a.raw_row = (long long)d->az_step * a.s_int * d->nbins;
    }
    if (d->sca) {
        // scatterometer mode: one channel, Kodis or Kirchhoff specular (the field scaled by
        // the two-way spreading like the Kodis field), Bragg model (hMTF, when on,
        // read at the rolled row of the [ny][field_nx] surface, unclipped); the columns are
        // whole range blocks of field_nx columns; the Bragg RCS is evaluated on every launch
        // and not stored
        if (d->nch != 1 || d->field_nx < 1 || d->nx % d->field_nx != 0 || d->roll < 0 || d->roll >= d->ny ||
            d->lut_block < 0)
            return OCS_ERR_ARG;
        a.lut_block = d->lut_d ? d->lut_block : 0;
        if (!(d->sr_bin_offset >= 0.0) || !(d->cap_t >= 0.0)) return OCS_ERR_ARG;
        if (d->nrcs_rows < 1 || d->nrcs_row < 0 || d->nrcs_row >= d->nrcs_rows) return OCS_ERR_ARG;
        a.sca = 1;
        a.az_f32 = d->az_f32 != 0;
        a.nblk = d->nx / d->field_nx;
        a.nrcs_row = d->nrcs_row;
        a.nrcs_rows = d->nrcs_rows;
        a.fnx = d->field_nx;
        a.roll = d->roll;
        a.sr_bin_off = d->sr_bin_offset;
        a.cap_t = d->cap_t;
        a.refresh = 1;
        a.scat = nullptr;
    } else {
        a.fnx = d->nx;
    }
    a.lut = d->lut_d;
    if (a.lut) {
        if (d->lut_naz < 1 || d->lut_ndy < 1 || d->lut_ndx < 1 || !(d->lut_daz != 0.0) || !(d->lut_ddy != 0.0) ||
            !(d->lut_ddx != 0.0))
            return OCS_ERR_ARG;
        a.lut_naz = d->lut_naz; a.lut_ndy = d->lut_ndy; a.lut_ndx = d->lut_ndx;
        a.lut_az0 = d->lut_az0; a.lut_daz = d->lut_daz; a.lut_dy0 = d->lut_dy0; a.lut_ddy = d->lut_ddy;
        a.lut_dx0 = d->lut_dx0; a.lut_ddx = d->lut_ddx;
    }
    return OCS_OK;
}

namespace ocs {

size_t pulse_args_bytes() { return sizeof(PulseArgs); }

int pulse_args_fill(const ocs_pulse_desc *d, void *out) {
    if (d && (d->sca || d->skim)) return OCS_ERR_ARG;   // the scene batch runs SAR scenes only
    PulseArgs a;
    const int st = fill_pulse_args(d, a);
    if (st != OCS_OK) return st;
    // The batch's scenes of these output groups have the local incidence's 1 - cos^2 from a
    // rounded square (one_minus_sq), the others from a fused one.  There is no physical ground
    // for it: the rule keeps the values that each group's scenes have always had.  The fused form
    // everywhere moves their NRCS sums, float64 totals of float32 cross sections, by up to 7e-9
    // (42 scenes at 20 to 44 degrees), while their error against float64 sections stays what it
    // is (9.4e-8 and 9.5e-8 at the scene that moves most).
    const int nout = a.npol * a.nch, w = width_class(nout < 4 ? nout : 4);
    const bool fast = a.do_kodis && a.do_bragg && a.npol == 1 && (nout >= 4 || nout == w) && !a.use_hmtf;
    a.rom.th_rounded = w == 2 ? (fast && !a.any_xti) : !fast;
    memcpy(out, &a, sizeof(a));
    return OCS_OK;
}

int batch_pulse_items(int nx, int ny, int tile_rows, int nout, int precision, int width) {
    const int G = precision == OCS_PREC_F64 ? 2 : 4;
    int groups = 0;
    for (int o = 0; o < nout; o += G) groups += width_class(nout - o < G ? nout - o : G) == width;
    return groups * ((nx + kPulseCols - 1) / kPulseCols) * ((ny + tile_rows - 1) / tile_rows);
}

int pulse_kind(const ocs_pulse_desc *d, int precision, int tile_rows) {
    if (d->do_kodis && d->spec_mode != 0) return kSlotKa;
    const double span = tile_span((double)d->facet_dx, d->inc_angle, d->binsize);
    const long long series = !d->do_bragg ? 0 : (d->n_m > d->n_p ? d->n_m : d->n_p);
    const bool grid = precision == OCS_PREC_MIXED ? mixed_hist_ok(d->nx, d->ny, series, span, d->binsize, tile_rows)
                                                  : f64_grid_ok(d->nx, d->ny, span);
    return grid ? kSlotStd : kSlotWide;
}

int batch_launch_pulse(const BatchRef &b, int precision, int kind, int width, int grid, cudaStream_t st) {
    if (grid < 1) return OCS_OK;
    if (kind != kSlotKa && precision == OCS_PREC_MIXED) return batch_pulse_split(b, kind, width, grid, st);
    if (kind == kSlotStd && precision == OCS_PREC_F64) return batch_pulse_f64(b, width, grid, st);
    return batch_pulse_general(b, precision, kind, width, grid, st);
}

}  // namespace ocs

extern "C" int64_t ocs_pulse_workspace_bytes(int32_t ny, int32_t nch) {
    if (ny < 1 || nch < 1 || nch > kMaxCh) return -1;
    return (int64_t)(mix_hdr_offset(ny, nch) + kMixHdrBytes);
}

// Whether the split-range mixed kernel takes this pulse: SAR mode with Kodis and / or
// direct / LUT Bragg scattering, the float32 scatterer series, column counts and base
// pointers that allow 16-byte bulk copies of every input row.
static bool mixed_split_ok(const ocs_pulse_desc *d);
namespace ocs {
bool pulse_split_ok(const ocs_pulse_desc *d) { return mixed_split_ok(d); }
}  // namespace ocs
static bool mixed_split_ok(const ocs_pulse_desc *d) {
    if (d->sca || d->skim || (d->do_kodis && d->spec_mode != 0) || !(d->do_kodis || d->do_bragg)) return false;
    if (d->do_bragg && (!d->s_m32_d || !d->s_p32_d)) return false;
    if (!d->diffx_d || !d->diffy_d || ((uintptr_t)d->rowtab_d & 15)) return false;
    return mix_inputs_ok(d);
}

// Compensation row of the mixed kernel (complex64 [npol*nch][nbins]) and the workspace
// header: reset before a scene (pending row -1, error flag 0, row zeroed).
extern "C" int ocs_pulse_reset(const ocs_pulse_desc *d, void *stream) {
    if (!d || !d->rowtab_d || d->ny < 1 || d->nch < 1 || d->nch > kMaxCh) return OCS_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    unsigned char *hdr = (unsigned char *)d->rowtab_d + mix_hdr_offset(d->ny, d->nch);
    if (cudaMemsetAsync(hdr, 0xff, 4, s) != cudaSuccess) return OCS_ERR_CUDA;
    if (cudaMemsetAsync(hdr + 4, 0, kMixHdrBytes - 4, s) != cudaSuccess) return OCS_ERR_CUDA;
    if (d->raw_lo_d) {
        const size_t n = (size_t)d->npol * d->nch * d->nbins * 2 * sizeof(float);
        if (cudaMemsetAsync(d->raw_lo_d, 0, n, s) != cudaSuccess) return OCS_ERR_CUDA;
    }
    return OCS_OK;
}

// Fold the last pulse's compensation row into its raw row (the scene's final step, or
// before the raw cube is read); no-op when nothing is pending.
extern "C" int ocs_pulse_flush(const ocs_pulse_desc *d, void *stream) {
    PulseArgs a;
    int st = fill_pulse_args(d, a);
    if (st != OCS_OK) return st;
    if (!d->raw_lo_d) return OCS_OK;
    const int nout = d->npol * d->nch;
    const long long n = (long long)nout * d->nbins;
    long long blocks = (n + 255) / 256;
    if (blocks > 1024) blocks = 1024;
    return launch_pdl(pulse_flush_kernel, dim3((unsigned)blocks), 256, 0, (cudaStream_t)stream, a, (float *)d->raw_lo_d, nout) ==
                   cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

// Status of the mixed kernel's bounded waits since the last reset (synchronises with the
// device): OCS_OK, or OCS_ERR_TIMEOUT if a wait gave up.
extern "C" int ocs_pulse_error(const ocs_pulse_desc *d) {
    if (!d || !d->rowtab_d || d->ny < 1 || d->nch < 1 || d->nch > kMaxCh) return OCS_ERR_ARG;
    int flag = 0;
    const unsigned char *hdr = (const unsigned char *)d->rowtab_d + mix_hdr_offset(d->ny, d->nch);
    if (cudaMemcpy(&flag, hdr + 4, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return OCS_ERR_CUDA;
    return flag ? OCS_ERR_TIMEOUT : OCS_OK;
}

// The launches that a pulse takes.  SAR pulses whose tiles fit the fine grid evaluate their rows
// themselves; the others run the register-window kernels behind a row-table launch.
struct PulseRoute {
    bool split, grid, refresh;
    int group;                              // outputs per pulse launch
    int hist_rows;                          // mixed fine grid: its tallest tiles, else 0
    bool row_table() const { return !grid; }
};

static PulseRoute pulse_route(const ocs_pulse_desc *d, const PulseArgs &a, int precision) {
    PulseRoute r;
    r.split = precision == OCS_PREC_MIXED && mixed_split_ok(d);
    // the fine grid folds the compensation row by complex64 vectors, the windows by floats
    const bool fold_ok = !d->raw_lo_d || !(((uintptr_t)d->raw_lo_d | (uintptr_t)d->raw_d) & 7);
    r.hist_rows = r.split && fold_ok ? split_hist_rows(a) : 0;
    r.grid = r.split ? r.hist_rows > 0
                     : precision == OCS_PREC_F64 && !a.sca && !a.skim && a.spec_mode == 0 &&
                           f64_grid_ok(a.nx, a.ny, tile_span(2.0 * a.kodis.hdx, a.inc_angle, a.binsize));
    r.refresh = a.refresh && a.do_bragg && !a.sca;
    r.group = precision == OCS_PREC_F64 && !r.grid ? 2 : 4;
    return r;
}

extern "C" int ocs_pulse_launches(const ocs_pulse_desc *d, int precision) {
    PulseArgs a;
    if (precision != OCS_PREC_F64 && precision != OCS_PREC_MIXED) return OCS_ERR_ARG;
    const int st = fill_pulse_args(d, a);
    if (st != OCS_OK) return st;
    const PulseRoute r = pulse_route(d, a, precision);
    return (r.refresh ? 1 : 0) + (r.row_table() ? 1 : 0) + (d->npol * d->nch + r.group - 1) / r.group;
}

extern "C" int ocs_pulse(const ocs_pulse_desc *d, int precision, void *stream) {
    PulseArgs a;
    int st = fill_pulse_args(d, a);
    if (st != OCS_OK) return st;
    if (precision != OCS_PREC_F64 && precision != OCS_PREC_MIXED) return OCS_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const int nout = d->npol * d->nch;
    const PulseRoute r = pulse_route(d, a, precision);
    float *lo_row = r.split ? (float *)d->raw_lo_d : nullptr;
    if (r.refresh) {
        st = launch_refresh(a, precision, s);
        if (st != OCS_OK) return st;
        a.refresh = 0;                      // the pulse kernels read the refreshed RCS
    }
    if (r.row_table() && r.split) {
        const int rows = d->ny > nout * d->nbins ? d->ny : nout * d->nbins;
        long long blocks = (rows + 127) / 128;
        if (blocks > 4096) blocks = 4096;
        pulse_rows_mixed_kernel<<<(unsigned)blocks, 128, 0, s>>>(a, lo_row, nout);
    } else if (r.row_table()) {
        pulse_rows_kernel<<<(d->ny + 127) / 128, 128, 0, s>>>(a);
    }
    if (cudaGetLastError() != cudaSuccess) return OCS_ERR_CUDA;
    MixMaps maps;
    if (r.split && !r.grid && !fill_mix_maps(d, maps)) return OCS_ERR_CUDA;
    for (int o = 0; o < nout; o += r.group) {
        a.out0 = o;
        a.nout = nout - o < r.group ? nout - o : r.group;
        st = r.split ? launch_pulse_split(a, maps, lo_row, r.hist_rows, s)
                     : (r.grid ? launch_pulse_f64(a, s) : launch_pulse_general(a, precision, s));
        if (st != OCS_OK) return st;
    }
    return OCS_OK;
}
