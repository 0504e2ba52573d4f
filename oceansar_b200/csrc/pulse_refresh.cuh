// Bragg RCS refresh (sar_raw_nompi.py:431-458): sqrt(RCS) of both Bragg lines of every facet
// from the Romeiser model (direct, or its LUT), and the pulse's NRCS sums.
//
// A pass of its own, one facet per thread, ahead of the refresh pulse's kernel, which then
// reads sqrt(RCS) like every other pulse.  The model is some 700 dependent instructions per
// facet and wants many resident warps, while the pulse kernels walk rows serially in few
// CTAs of many registers: inside them a refresh cost 216 us more than an ordinary pulse
// on 2048^2 facets (mixed), and 51 us on 256^2; as a pass it costs what the model costs.
#pragma once
#include "pulse_core.cuh"

namespace ocs {

constexpr int kRefCols = 128;       // columns (threads) of an item

OCS_HD int refresh_items(int nx, int ny, int rows) { return ((nx + kRefCols - 1) / kRefCols) * ((ny + rows - 1) / rows); }
// Rows of an item: enough to share the rows' azimuth set-up, few on small surfaces, which
// need every item to fill the GPU.  A refresh with one row and with four: 256^2 5.9 and 12.8 us
// (float64 5.9 and 17.8), 900^2 41.6 and 39.7 (75.4 and 76.4), 1024^2 47.4 and 42.6 (86.8 and 77.9),
// 2048^2 184 and 154 (341 and 306).
OCS_HD int refresh_rows(int nx, int ny) { return (long long)nx * ny >= (1 << 20) ? 4 : 1; }

// One item of kRefCols columns x `rows` (<= 4) rows; every thread of a kRefCols CTA calls it.
template <typename T>
OCS_D void refresh_item(const PulseArgs &a, double az_now, int az_step, int item, int rows) {
    __shared__ double srow[4][3];               // azimuth angle, its cos and sin
    __shared__ double sred[32];
    const int tiles_x = (a.nx + kRefCols - 1) / kRefCols;
    const int x = (item % tiles_x) * kRefCols + threadIdx.x;
    const int y0 = (item / tiles_x) * rows, n = min(rows, a.ny - y0);
    __syncthreads();
    if ((int)threadIdx.x < n) {
        const double azp = asin(dsub((double)a.y[y0 + threadIdx.x], az_now) / a.gr0);
        srow[threadIdx.x][0] = azp;
        srow[threadIdx.x][1] = cos(azp);
        srow[threadIdx.x][2] = sin(azp);
    }
    __syncthreads();
    double sum[2] = {0.0, 0.0};
    if (x < a.nx) {
        const T inc = (T)a.inc[x];
        const long long npix = (long long)a.nx * a.ny;
        T *scat = reinterpret_cast<T *>(a.scat);
        for (int r = 0; r < n; ++r) {
            const long long idx = (long long)(y0 + r) * a.nx + x;
            const float dx = a.diffx[idx], dy = a.diffy[idx];
            T hh[2], vv[2];
            if (a.lut) {
                // the table holds the model's output polarisation(s) in output order
                const int ai = lut_az_index(a, srow[r][0]);
                T r0[2], r1[2];
                romeiser_lut<T>(a, ai, dx, dy, 0, r0);
                if (a.npol == 2) romeiser_lut<T>(a, ai, dx, dy, 1, r1);
                else { r1[0] = r0[0]; r1[1] = r0[1]; }
                const bool vv_first = a.rom.pol == POL_VV;
                hh[0] = vv_first ? r1[0] : r0[0]; hh[1] = vv_first ? r1[1] : r0[1];
                vv[0] = vv_first ? r0[0] : r1[0]; vv[1] = vv_first ? r0[1] : r1[1];
            } else {
                romeiser_facet<T>(a.rom, inc, (T)srow[r][0], (T)srow[r][1], (T)srow[r][2], (T)dx, (T)dy, hh, vv);
            }
            if (a.use_hmtf) {
                float hm = a.hmtf[idx];
                hm = hm < -1.f ? -1.f : hm;
                const T f = (T)(1.f + hm);
                hh[0] *= f; hh[1] *= f; vv[0] *= f; vv[1] *= f;
            }
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                if (p < a.npol) {
                    const bool use_vv = a.rom.pol == POL_VV || (a.rom.pol == POL_DP && p == 1);
                    const T r0 = use_vv ? vv[0] : hh[0], r1 = use_vv ? vv[1] : hh[1];
                    sum[p] += (double)r0 + (double)r1;
                    scat[(2 * p) * npix + idx] = tsqrt(r0);
                    scat[(2 * p + 1) * npix + idx] = tsqrt(r1);
                }
            }
        }
    }
    for (int p = 0; p < a.npol; ++p)
        block_atomic_sum(sum[p], &a.nrcs_bragg[(long long)p * a.az_steps + az_step], sred);
}

int launch_refresh(const PulseArgs &a, int precision, cudaStream_t st);

}  // namespace ocs
