// Standalone facet-to-range-bin accumulation: the drop-in for chan_profile_numba
// (oceansar/radarsim/range_profile.py:83-116 -> profile_integrator :22-49 and
// profile_integrator_1d :52-80).
//
// Facets come in arbitrary order (the caller's flattened slant-range / scene arrays), so
// each thread takes a run of consecutive facets -- consecutive facets of a flattened
// surface row are consecutive ground-range columns, whose bins grow monotonically -- and
// accumulates them through the register window of accum.cuh.  Facets that keep their
// [ny][nx] surface shape go through the fine-grid kernel below (one shared-memory add per
// facet into a (bin, LUT index) histogram, convolved with the pulse once per tile).  Output
// is accumulated in place (+=), never cleared, exactly like the reference.
#include <string.h>

#include "accum.cuh"

namespace ocs {

constexpr int kProfThreads = 256;

// Dynamic shared memory layout: [wtab | CTA bin accumulator].
template <typename T, int S>
__global__ void __launch_bounds__(kProfThreads)
chan_profile_kernel(const double *__restrict__ srg, const cplx<T> *__restrict__ scene,
                    long long npts, long long row_len, double binsize, double min_sr,
                    const float *__restrict__ sinc, int taps, int ovs, T *__restrict__ out,
                    int nbins, long long out_row_stride, int chunk, int cta_nbw) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *wtab = reinterpret_cast<T *>(smem_raw);
    const int wlen = wtab_len<T, S>(taps, ovs);
    T *acc = wtab + ((wlen + 3) & ~3);

    // Row handling (profile_integrator_1d): facets of row r accumulate into out row r.
    // A CTA covers facets [f0, f0 + blockDim*chunk) of one row.
    const long long ctas_per_row = (row_len + (long long)kProfThreads * chunk - 1) /
                                   ((long long)kProfThreads * chunk);
    const long long row = blockIdx.x / ctas_per_row;
    const long long f0 = row * row_len + (blockIdx.x % ctas_per_row) * (long long)kProfThreads * chunk;
    const long long fend = min(row * row_len + row_len, npts);
    if (f0 >= fend) return;

    build_wtab<T, S>(wtab, sinc, taps, ovs);

    CtaBins<T, 1> cb;
    cb.acc = acc;
    cb.nbw = cta_nbw;
    cb.nout = 1;
    cb.nbins = nbins;
    cb.out = out + 2 * row * out_row_stride;
    cb.out_stride = 0;
    if (cta_nbw >= nbins) {
        cb.cta_base = 0;
    } else {
        int b0, l0;
        bin_and_lut(srg[f0], min_sr, binsize, ovs, b0, l0);
        cb.cta_base = b0 - cta_nbw / 2;
    }
    cb.zero();
    __syncthreads();

    BinWindow<T, S, 1> win;
    win.reset();
    const int half = taps / 2;
    const long long my0 = f0 + (long long)threadIdx.x * chunk;
    for (int k = 0; k < chunk; ++k) {
        long long i = my0 + k;
        if (i >= fend) break;
        int bin_d, lut;
        bin_and_lut(srg[i], min_sr, binsize, ovs, bin_d, lut);
        if (bin_d < -(1 << 29)) continue;
        cplx<T> c[1] = {scene[i]};
        win.add(bin_d - half, lut, c, wtab, sinc, taps, ovs, cb);
    }
    win.flush(cb);
    __syncthreads();
    cb.flush_to_global();
}

template <typename T, int S>
static int launch_chan_profile(const double *srg, const void *scene, long long naz, long long npts,
                               double binsize, double min_sr, const float *sinc, int taps, int ovs,
                               T *out, int nbins, cudaStream_t stream) {
    if (taps < 1 || taps > S || ovs < 1 || npts < 0 || naz < 1 || nbins < 0) return OCS_ERR_ARG;
    if (npts == 0 || nbins == 0) return OCS_OK;
    const int wlen = wtab_len<T, S>(taps, ovs);
    const size_t wtab_bytes = (size_t)((wlen + 3) & ~3) * sizeof(T);
    const size_t budget = 96 * 1024;
    if (wtab_bytes > budget / 2) return OCS_ERR_UNSUPPORTED;
    long long cap = (long long)((budget - wtab_bytes) / (2 * sizeof(T)));
    int nbw = (int)(nbins < cap ? nbins : cap);
    if (nbw > 8192) nbw = 8192;
    // Enough CTAs to fill the GPU, but long enough runs per thread to keep the windows warm.
    long long total = naz * npts;
    long long ch = total / (148LL * 8 * kProfThreads);
    int chunk = (int)(ch < 1 ? 1 : (ch > 32 ? 32 : ch));
    long long ctas_per_row = (npts + (long long)kProfThreads * chunk - 1) / ((long long)kProfThreads * chunk);
    long long grid = ctas_per_row * naz;
    if (grid > 0x7fffffffLL) return OCS_ERR_SIZE;
    size_t smem = wtab_bytes + (size_t)nbw * 2 * sizeof(T);
    auto kern = chan_profile_kernel<T, S>;
    if (ensure_smem((const void *)kern, smem) != cudaSuccess)
        return OCS_ERR_CUDA;
    kern<<<(unsigned)grid, kProfThreads, smem, stream>>>(
        srg, reinterpret_cast<const cplx<T> *>(scene), naz * npts, npts, binsize, min_sr, sinc, taps,
        ovs, out, nbins, (long long)nbins, chunk, nbw);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

// Scene value of one facet: one vector load when the scene is aligned to its element pair.
template <typename T, bool VEC> OCS_D cplx<T> load_scene(const cplx<T> *p) {
    if constexpr (VEC) {
        if constexpr (sizeof(T) == 4) {
            const float2 v = __ldg(reinterpret_cast<const float2 *>(p));
            return {v.x, v.y};
        } else {
            const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
            return {v.x, v.y};
        }
    } else {
        return {__ldg(&p->re), __ldg(&p->im)};
    }
}

// ---------------------------------------------------------------------------------------
// Flattened facet list through a fine grid.
//
// What bounded the run-per-thread kernel above (0.11 of the copy rate):
// every thread reads a run of its own, so a warp's loads touch 32 lines; windows of 16 bins in
// 127 registers leave 16 warps per SM; neighbouring lanes flush them to the same shared bins
// one after the other.  Here a CTA of 1024 threads walks its part of the list with coalesced
// loads, four facets per thread in flight, and adds each facet once to a shared grid H of (bin,
// LUT index) cells (see the two-dimensional form below), HB bins wide, convolved with the pulse
// at the end.  H is placed over the bins of the first facets.  If others lie outside, further
// passes over the part, one per window of HB bins that holds any, take them: they read the
// ranges again, from the L2 cache, and the scene values of their own facets only.  Parts that
// would take more than flat_windows passes (lists in random order, or rows wider than H, over
// many bins) add each facet's taps to shared output bins instead, in one pass.
// Measured, ranges and values read from memory (L2 flushed), f64, run-per-thread kernel -> grid:
// 3 M facets sorted by range over 4096 bins 293 -> 113 us; rows 450 bins wide 106 -> 43; in random
// order over 512 bins 262 -> 45; over 4096 bins, where taps take over, 270 -> 168; 100 k facets of
// rows 3700 bins wide 27 -> 16 (windows alone 66); 10 k in random order 14 -> 18.
// Sorted lists of more than some 6 M facets, whose lanes all add to the same few cells, were faster
// by runs (12 M over 512 bins 494 -> 688).
// H and the output bins are float64 for both element types: a cell may sum thousands of facets.
constexpr int kFlatThreads = 1024;
constexpr int kFlatPer = 4;                  // facets per thread in flight
constexpr int kFlatMaxHB = 512;
constexpr int kFlatMaxWindows = 24;          // windows of HB bins the output may take
constexpr size_t kFlatGridBytes = 200 * 1024;
static_assert((size_t)kFlatMaxWindows * kFlatMaxHB * 2 * sizeof(double) <= kFlatGridBytes, "output bins of a part");

// Further windows that a part of `chunk` facets may take before its facets go tap by tap.
// A window costs a pass over the part's ranges and its share of H's clearing and convolution, the
// taps sixteen shared adds per facet instead of two: 676 facets 8 us a window, taps 4 us; 6757
// facets two windows 59 us, taps 68, three 80 and 68; 20 k facets three windows 125, taps 172,
// seven 213 and 168; 81 k facets seven 762 and 614 (random order; float64).
OCS_D int flat_windows(long long chunk) { return chunk < 4096 ? 0 : (int)min(6LL, 2 + chunk / 8192); }

template <typename T> OCS_D void flat_add_out(T *out, int nbins, int b, T re, T im) {
    if (b < 0 || b >= nbins) return;
    atomicAdd(out + 2 * (long long)b, re);
    atomicAdd(out + 2 * (long long)b + 1, im);
}

// Non-finite values: exactly their own taps.
template <typename T> OCS_D void flat_own_taps(const T *w, int taps, int L, int b, int l, cplx<T> c, T *out, int nbins) {
    for (int j = 0; j < taps; ++j) {
        const T wj = w[j * L + l];
        flat_add_out(out, nbins, b - taps / 2 + j, wj * c.re - (T)0 * c.im, wj * c.im + (T)0 * c.re);
    }
}

// Every facet of [f0, f1) whose bin lies in [lo, hi] but not in [wb, wb + HB), tap by tap, through
// the output bins that they reach, in shared memory (B, the place of H).
template <typename T, bool VEC, class Acc>
__device__ __noinline__ void flat_by_taps(const double *__restrict__ srg, const cplx<T> *__restrict__ scene, long long f0,
                                          long long f1, double binsize, double inv_binsize, double min_sr, const T *w,
                                          Acc *B, int taps, int ovs, T *__restrict__ out, int nbins, int lo, int hi,
                                          int wb, int HB) {
    const int t = threadIdx.x, L = ovs + 1, half = taps / 2;
    const int o0 = max(lo - half, 0), o1 = min(hi - half + taps, nbins);
    __syncthreads();                         // H has been read
    for (int i = t; i < 2 * (o1 - o0); i += kFlatThreads) B[i] = (Acc)0;
    __syncthreads();
    for (long long i0 = f0 + t; i0 < f1; i0 += kFlatPer * kFlatThreads) {
        double s[kFlatPer];
        cplx<T> c[kFlatPer];
#pragma unroll
        for (int u = 0; u < kFlatPer; ++u) {
            const long long i = i0 + u * kFlatThreads;
            if (i < f1) {
                s[u] = __ldg(srg + i);
                c[u] = load_scene<T, VEC>(scene + i);
            }
        }
#pragma unroll
        for (int u = 0; u < kFlatPer; ++u) {
            const long long i = i0 + u * kFlatThreads;
            if (i >= f1) continue;
            int b, l;
            bin_lut_magic(div_by(dsub(s[u], min_sr), binsize, inv_binsize), (double)ovs, b, l);
            if (b < lo || b > hi || (unsigned)(b - wb) < (unsigned)HB) continue;
            if (!isfinite(c[u].re + c[u].im)) {
                flat_own_taps(w, taps, L, b, l, c[u], out, nbins);
                continue;
            }
            for (int j = 0; j < taps; ++j) {
                const int o = b - half + j;
                if (o < 0 || o >= nbins) continue;
                const Acc wj = (Acc)w[j * L + l];
                atomicAdd(B + 2 * (o - o0), wj * (Acc)c[u].re);
                atomicAdd(B + 2 * (o - o0) + 1, wj * (Acc)c[u].im);
            }
        }
    }
    __syncthreads();
    for (int i = t; i < 2 * (o1 - o0); i += kFlatThreads)
        if (B[i] != (Acc)0) atomicAdd(out + 2 * (long long)o0 + i, (T)B[i]);
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kFlatThreads, 1)
chan_profile_flat_kernel(const double *__restrict__ srg, const cplx<T> *__restrict__ scene, long long npts,
                         double binsize, double inv_binsize, double min_sr, const float *__restrict__ sinc, int taps,
                         int ovs, T *__restrict__ out, int nbins, long long chunk, int HB, unsigned grid_bytes) {
    using Acc = double;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_lo, s_hi;
    const int L = ovs + 1, t = threadIdx.x;
    Acc *Hre = reinterpret_cast<Acc *>(smem_raw), *Him = Hre + HB * L;
    T *w = reinterpret_cast<T *>(smem_raw + grid_bytes);                  // [taps][L]
    const long long f0 = blockIdx.x * chunk, f1 = min(f0 + chunk, npts);
    const int half = taps / 2;
    // facets that reach a valid output bin have their own bin in [first, last]
    const int first = half - taps + 1, last = nbins - 1 + half;
    auto bin_of = [&](double s, int &b, int &l) {
        bin_lut_magic(div_by(dsub(s, min_sr), binsize, inv_binsize), (double)ovs, b, l);
    };
    auto block_range = [&](int lo, int hi, int &blo, int &bhi) {
        __syncthreads();
        if (t == 0) { s_lo = 0x7fffffff; s_hi = -0x7fffffff; }
        __syncthreads();
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if ((t & 31) == 0) { atomicMin(&s_lo, lo); atomicMax(&s_hi, hi); }
        __syncthreads();
        blo = s_lo;
        bhi = s_hi;
    };
    auto by_taps = [&](int lo, int hi, int wb) {
        flat_by_taps<T, VEC>(srg, scene, f0, f1, binsize, inv_binsize, min_sr, w, Hre, taps, ovs, out, nbins, lo, hi, wb, HB);
    };
    int base;                                // first bin of window 0
    {
        int lo = 0x7fffffff, hi = -0x7fffffff;
#pragma unroll
        for (int k = 0; k < kFlatPer; ++k) {
            const long long i = f0 + t + k * kFlatThreads;
            int b, l;
            if (i >= f1) continue;
            bin_of(__ldg(srg + i), b, l);
            if (b >= first && b <= last) { lo = min(lo, b); hi = max(hi, b); }
        }
        for (int i = t; i < taps * L; i += kFlatThreads) w[i] = (T)sinc[i % L + (i / L) * ovs];
        int blo, bhi;
        block_range(lo, hi, blo, bhi);
        if (blo <= bhi && bhi - blo >= (1 + flat_windows(chunk)) * HB) {
            by_taps(first, last, last + 1);
            return;
        }
        base = bhi < blo ? first : (bhi - blo < HB ? blo - (HB - (bhi - blo + 1)) / 2 : blo - 8);
    }
    int kmin = 0, kmax = 0;                  // windows base + k HB that hold facets
    for (int k = 0, pass = 0;; ++pass) {
        for (int i = t; i < 2 * HB * L; i += kFlatThreads) Hre[i] = (Acc)0;
        __syncthreads();
        const int wb = base + k * HB;        // first bin of this pass's window
        int tlo = HB, thi = -1, mlo = 0x7fffffff, mhi = -0x7fffffff;
        for (long long i0 = f0 + t; i0 < f1; i0 += kFlatPer * kFlatThreads) {
            double s[kFlatPer];
            cplx<T> c[kFlatPer];
#pragma unroll
            for (int u = 0; u < kFlatPer; ++u) {
                const long long i = i0 + u * kFlatThreads;
                if (i < f1) {
                    s[u] = __ldg(srg + i);
                    if (pass == 0) c[u] = load_scene<T, VEC>(scene + i);
                }
            }
#pragma unroll
            for (int u = 0; u < kFlatPer; ++u) {
                const long long i = i0 + u * kFlatThreads;
                if (i >= f1) continue;
                int b, l;
                bin_of(s[u], b, l);
                if (b < first || b > last) continue;          // no valid tap (invalid ranges among them)
                const int r = b - wb;
                if ((unsigned)r >= (unsigned)HB) {
                    mlo = min(mlo, b);
                    mhi = max(mhi, b);
                    continue;
                }
                if (pass > 0) c[u] = load_scene<T, VEC>(scene + i);
                if (!isfinite(c[u].re + c[u].im)) {
                    flat_own_taps(w, taps, L, b, l, c[u], out, nbins);
                    continue;
                }
                atomicAdd(Hre + r * L + l, (Acc)c[u].re);
                atomicAdd(Him + r * L + l, (Acc)c[u].im);
                tlo = min(tlo, r);
                thi = max(thi, r);
            }
        }
        int clo, chi, olo = 0, ohi = -1;
        if (pass == 0) {
            // windows of the facets outside window 0 (floor division)
            block_range(mlo, mhi, olo, ohi);
            if (olo <= ohi) {
                if (olo < base) kmin = -((base - olo + HB - 1) / HB);
                if (ohi >= base + HB) kmax = (ohi - base) / HB;
            }
        }
        block_range(tlo, thi, clo, chi);     // (its barriers complete H)
        // convolve the touched rows with the pulse: four lanes per output bin, a quarter of the
        // taps each
        const int items = chi < clo ? 0 : (chi - clo + taps) * 4, tq = (taps + 3) / 4, q = t & 3;
        for (int i0 = 0; i0 < items; i0 += kFlatThreads) {
            const int i = i0 + t, m = i >> 2;
            Acc sre = (Acc)0, sim = (Acc)0;
            if (i < items) {
                for (int j = q * tq; j < min(taps, (q + 1) * tq); ++j) {
                    const int r = clo + m - j;
                    if (r < clo || r > chi) continue;
                    for (int l = 0; l < L; ++l) {
                        const Acc wl = (Acc)w[j * L + l];
                        sre = fma(wl, Hre[r * L + l], sre);
                        sim = fma(wl, Him[r * L + l], sim);
                    }
                }
            }
            sre += __shfl_xor_sync(0xffffffffu, sre, 1);
            sim += __shfl_xor_sync(0xffffffffu, sim, 1);
            sre += __shfl_xor_sync(0xffffffffu, sre, 2);
            sim += __shfl_xor_sync(0xffffffffu, sim, 2);
            if (i < items && q == 0 && (sre != (Acc)0 || sim != (Acc)0)) flat_add_out(out, nbins, wb + clo - half + m, (T)sre, (T)sim);
        }
        if (kmax - kmin > flat_windows(chunk)) {        // (decided in pass 0)
            by_taps(olo, ohi, base);
            return;
        }
        // next window that may hold facets: kmin .. kmax without 0
        k = pass == 0 ? kmin : k + 1;
        if (k == 0) ++k;
        if (k > kmax) break;
        __syncthreads();                     // H is read before it is cleared
    }
}

// Bins of the grid for a list, 0 where the run-per-thread kernel takes it: oversampling so fine
// that H holds few bins, outputs of more bins than shared memory holds, or a divisor whose reciprocal
// is no normal number.
template <typename T> static int flat_grid_bins(int taps, int ovs, double binsize, int nbins) {
    if (taps < 1 || taps > 16 || ovs < 1 || ovs > 1024 || !(fabs(binsize) > 1e-100 && fabs(binsize) < 1e100)) return 0;
    long long hb = (long long)(kFlatGridBytes / (2 * sizeof(T) * (ovs + 1)));
    if (hb > kFlatMaxHB) hb = kFlatMaxHB;
    if (hb < 64 || nbins > kFlatMaxWindows * hb) return 0;
    hb = (long long)(kFlatGridBytes / (2 * sizeof(double) * (ovs + 1)));
    return hb > kFlatMaxHB ? kFlatMaxHB : (int)hb;
}

template <typename T>
static int launch_chan_profile_flat(const double *srg, const void *scene, long long npts, double binsize, double min_sr,
                                    const float *sinc, int taps, int ovs, T *out, int nbins, int HB, cudaStream_t st) {
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return OCS_ERR_CUDA;
    // H, or the output bins that take its place
    size_t grid_bytes = 2 * sizeof(double) * (HB * (ovs + 1) > nbins ? HB * (ovs + 1) : nbins);
    grid_bytes = (grid_bytes + 15) & ~(size_t)15;
    const size_t smem = grid_bytes + (size_t)taps * (ovs + 1) * sizeof(T);
    long long ctas = (npts + kFlatThreads - 1) / kFlatThreads;
    if (ctas > sms) ctas = sms;
    const long long chunk = (npts + ctas - 1) / ctas;
    ctas = (npts + chunk - 1) / chunk;
    const bool vec = ((uintptr_t)scene & (2 * sizeof(T) - 1)) == 0;
    auto k = vec ? chan_profile_flat_kernel<T, true> : chan_profile_flat_kernel<T, false>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    k<<<(unsigned)ctas, kFlatThreads, smem, st>>>(srg, reinterpret_cast<const cplx<T> *>(scene), npts, binsize,
                                                  1.0 / binsize, min_sr, sinc, taps, ovs, out, nbins, chunk, HB,
                                                  (unsigned)grid_bytes);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

// ---------------------------------------------------------------------------------------
// Two-dimensional layout: the facets are a [ny][nx] surface (rows = azimuth, columns =
// ground range), as sar_raw flattens them.  A CTA takes tiles of kC2Cols columns x up to
// kC2Rows rows; a thread owns one column and walks down the rows, so a warp reads 32
// consecutive facets of a row (coalesced) and every thread's range bin drifts only with
// the azimuth curvature and the surface displacement -- its register window almost never
// moves.
constexpr int kC2Cols = 128;
constexpr int kC2Rows = 64;
constexpr int kC2Nbw = 256;

// Register-batched form of the two-dimensional accumulation: persistent CTAs walk tiles
// of kC2Cols columns x tile_rows rows; every thread loads the slant ranges and scene
// values of its column for kRB rows at once (2 kRB independent coalesced loads in flight
// per thread) and then runs them through its register window.  The kernel is bound by
// the latency of each facet's dependent chain (bin -> weight row -> multiply-adds), so
// resident warps count most: single precision runs 4-row batches at 6 CTAs per SM
// (within 80 registers), float64 8-row batches at 4 (its window takes twice the registers).
template <typename T> __host__ __device__ constexpr int rows_per_batch() { return sizeof(T) == 4 ? 4 : 8; }
template <typename T> __host__ __device__ constexpr int ctas_per_sm_2d() { return sizeof(T) == 4 ? 6 : 4; }

template <typename T, int S>
__global__ void __launch_bounds__(kC2Cols, ctas_per_sm_2d<T>())
chan_profile_2d_regs_kernel(const double *__restrict__ srg, const cplx<T> *__restrict__ scene, int ny, int nx,
                            double binsize, double min_sr, const float *__restrict__ sinc, int taps, int ovs,
                            T *__restrict__ out, int nbins, int tile_rows) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *wtab = reinterpret_cast<T *>(smem_raw);
    const int wlen = wtab_len<T, S>(taps, ovs);
    T *acc = wtab + ((wlen + 3) & ~3);
    build_wtab<T, S>(wtab, sinc, taps, ovs);
    const int tiles_x = (nx + kC2Cols - 1) / kC2Cols;
    const int tiles = tiles_x * ((ny + tile_rows - 1) / tile_rows);
    const double inv_binsize = 1.0 / binsize;
    const int half = taps / 2;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int x0 = (tile % tiles_x) * kC2Cols;
        const int y0 = (tile / tiles_x) * tile_rows;
        const int nrows = min(tile_rows, ny - y0);
        const int x = x0 + threadIdx.x;
        __syncthreads();                  // the previous tile's bins are flushed (and wtab built)
        CtaBins<T, 1> cb;
        cb.acc = acc;
        cb.nbw = kC2Nbw;
        cb.nout = 1;
        cb.nbins = nbins;
        cb.out = out;
        cb.out_stride = 0;
        {
            int b0, l0;
            bin_and_lut(srg[(long long)y0 * nx + x0], min_sr, binsize, ovs, b0, l0);
            cb.cta_base = (b0 > -(1 << 29)) ? b0 - kC2Nbw / 4 : 0;
        }
        cb.zero();
        __syncthreads();
        BinWindow<T, S, 1> win;
        win.reset();
        if (x < nx) {
            const long long g0 = (long long)y0 * nx + x;
            constexpr int kRB = rows_per_batch<T>();
            for (int i0 = 0; i0 < nrows; i0 += kRB) {
                double sr[kRB];
                cplx<T> c[kRB];
#pragma unroll
                for (int k = 0; k < kRB; ++k) {
                    if (i0 + k < nrows) {
                        const long long g = g0 + (long long)(i0 + k) * nx;
                        sr[k] = __ldg(srg + g);
                        c[k] = scene[g];
                    }
                }
#pragma unroll
                for (int k = 0; k < kRB; ++k) {
                    if (i0 + k >= nrows) break;
                    int bin_d, lut;
                    // FP64: IEEE division, bin / LUT bit-identical with numpy; single
                    // precision: reciprocal multiply (a one-ulp difference in the bin coordinate)
                    if (sizeof(T) == 8) bin_and_lut(sr[k], min_sr, binsize, ovs, bin_d, lut);
                    else bin_and_lut_fast(sr[k], min_sr, inv_binsize, ovs, bin_d, lut);
                    if (bin_d < -(1 << 29)) continue;
                    cplx<T> cc[1] = {c[k]};
                    win.add(bin_d - half, lut, cc, wtab, sinc, taps, ovs, cb);
                }
            }
        }
        win.flush(cb);
        __syncthreads();
        cb.flush_to_global();
    }
}

template <typename T, int S>
static int launch_chan_profile_2d_regs(const double *srg, const void *scene, long long ny, long long nx,
                                       double binsize, double min_sr, const float *sinc, int taps, int ovs, T *out,
                                       int nbins, cudaStream_t stream) {
    if (taps < 1 || taps > S || ovs < 1) return OCS_ERR_ARG;
    if (ny > 0x7fffffffLL || nx > 0x7fffffffLL) return OCS_ERR_SIZE;
    const int wlen = wtab_len<T, S>(taps, ovs);
    const size_t smem = (size_t)((wlen + 3) & ~3) * sizeof(T) + (size_t)kC2Nbw * 2 * sizeof(T);
    auto kern = chan_profile_2d_regs_kernel<T, S>;
    if (ensure_smem((const void *)kern, smem) != cudaSuccess) return OCS_ERR_CUDA;
    const int resident = resident_ctas((const void *)kern, kC2Cols, smem);
    if (resident <= 0) return OCS_ERR_CUDA;
    const long long tiles_x = (nx + kC2Cols - 1) / kC2Cols;
    const long long want = (long long)resident * ((tiles_x * ((ny + kC2Rows - 1) / kC2Rows) + resident - 1) / resident);
    long long per_col = want / tiles_x;
    if (per_col < 1) per_col = 1;
    long long rows = (ny + per_col - 1) / per_col;
    rows = rows < 8 ? (ny < 8 ? ny : 8) : (rows > kC2Rows ? kC2Rows : rows);
    const long long tiles = tiles_x * ((ny + rows - 1) / rows);
    const long long grid = tiles < resident ? tiles : resident;
    kern<<<(unsigned)grid, kC2Cols, smem, stream>>>(srg, reinterpret_cast<const cplx<T> *>(scene), (int)ny, (int)nx,
                                                      binsize, min_sr, sinc, taps, ovs, out, nbins, (int)rows);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

// ---------------------------------------------------------------------------------------
// Fine-grid form of the two-dimensional accumulation.  A facet's taps depend only on its
// range bin and LUT index, so with H[bin][l] = the sum of the coefficients of the facets
// whose bin is `bin` and whose LUT index is l,
//     out[b] = sum over facets of sinc[lut + j ovs] c,  j = b - (bin - taps/2)
//            = sum_{j < taps} sum_{l <= ovs} sinc[l + j ovs] H[b + taps/2 - j][l].
// A CTA adds each facet's coefficient once into a shared-memory H that spans kHB bins
// around its tile of 128 columns x tile_rows rows (two shared atomic adds per facet into
// separate real and imaginary planes, instead of a multiply-add per tap and window slot; no
// register window, so 8 to 12 CTAs fit per SM), then convolves H with the oversampled pulse
// once per tile and adds the result to the output with global atomics.  A tile whose first
// and last rows span more bins than H holds is walked in narrower column groups (64 or 32
// columns, two or four rows per step, one H each); facets whose bin still falls outside H,
// and facets with non-finite coefficients (which must touch exactly their own taps, with
// the reference's complex product), take the direct path of per-tap global atomics.  Bins
// outside [0, nbins) are dropped, as the reference's edge branch does.
constexpr int kHThreads = 128;
constexpr int kHRB = 4;             // rows of loads in flight per thread
constexpr int kHB = 64;             // bins held by H
// Resident CTAs per SM: single precision fits twelve within 40 registers; float64 keeps
// eight (its division and 16-byte loads need the registers).
template <typename T> __host__ __device__ constexpr int hist_ctas_per_sm() { return sizeof(T) == 4 ? 12 : 8; }

template <typename T>
OCS_D void direct_taps(int bin_d, int lut, cplx<T> c, const float *sinc, int taps, int ovs, T *out, int nbins) {
    const int first = bin_d - taps / 2;
    for (int j = 0; j < taps; ++j) {
        const int b = first + j;
        if (b < 0 || b >= nbins) continue;
        const T w = (T)sinc[lut + j * ovs];
        atomicAdd(out + 2 * b, w * c.re - (T)0 * c.im);
        atomicAdd(out + 2 * b + 1, w * c.im + (T)0 * c.re);
    }
}

template <typename T> OCS_HD size_t hist_smem_bytes(int taps, int ovs) {
    return (((size_t)taps * (ovs + 1) * sizeof(T) + 15) & ~(size_t)15) + (size_t)kHB * (ovs + 1) * sizeof(cplx<T>) +
           16 * sizeof(int);
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kHThreads, hist_ctas_per_sm<T>())
chan_profile_2d_hist_kernel(const double *__restrict__ srg, const cplx<T> *__restrict__ scene, int ny, int nx,
                            double binsize, double min_sr, const float *__restrict__ sinc, int taps, int ovs,
                            T *__restrict__ out, int nbins, int tile_rows) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int L = ovs + 1;
    T *w = reinterpret_cast<T *>(smem_raw);                                   // [taps][L]
    // H as two planes (real, imaginary) of [kHB][L]: the lanes of one atomic add spread
    // over all 32 banks
    T *Hre = reinterpret_cast<T *>(smem_raw + (((size_t)taps * L * sizeof(T) + 15) & ~(size_t)15));
    T *Him = Hre + kHB * L;
    int *s_lo = reinterpret_cast<int *>(Him + kHB * L);                       // [4] per-warp bin estimates
    int *s_hi = s_lo + 4;
    int *s_tlo = s_lo + 8;                                                    // [4] per-warp touched cells
    int *s_thi = s_lo + 12;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < taps * L; i += kHThreads) {
        const int j = i / L, l = i - j * L;
        w[i] = (T)sinc[l + j * ovs];
    }
    const int tiles_x = (nx + kHThreads - 1) / kHThreads;
    const int tiles = tiles_x * ((ny + tile_rows - 1) / tile_rows);
    const double inv_binsize = 1.0 / binsize;
    const double dovs = (double)ovs;
    const int half = taps / 2;
    auto bin_of = [&](double s, int &bin_d, int &lut) {
        // float64: IEEE division (bins and LUT indices bit-identical with numpy); single
        // precision: reciprocal multiply (a one-ulp difference in the bin coordinate)
        const double bin_f = sizeof(T) == 8 ? ddiv(dsub(s, min_sr), binsize) : (s - min_sr) * inv_binsize;
        bin_lut_magic(bin_f, dovs, bin_d, lut);
    };
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int x0 = (tile % tiles_x) * kHThreads;
        const int y0 = (tile / tiles_x) * tile_rows;
        const int nrows = min(tile_rows, ny - y0);
        __syncthreads();                  // the previous tile's convolution has read H (and w is built)
        // ---- bins of the tile's first and last rows, per warp of 32 columns ----
        {
            int lo = 0x3fffffff, hi = -0x3fffffff;
            const int x = x0 + t;
            if (x < nx) {
                int b, l;
                bin_of(__ldg(srg + (long long)y0 * nx + x), b, l);
                if (b > -(1 << 29)) { lo = min(lo, b); hi = max(hi, b); }
                bin_of(__ldg(srg + (long long)(y0 + nrows - 1) * nx + x), b, l);
                if (b > -(1 << 29)) { lo = min(lo, b); hi = max(hi, b); }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if (lane == 0) { s_lo[warp] = lo; s_hi[warp] = hi; }
        }
        for (int i = t; i < kHB * L; i += kHThreads) { Hre[i] = (T)0; Him[i] = (T)0; }
        __syncthreads();
        // column groups: 128 columns when the tile's bins fit H with room for the jitter
        // between its first and last rows, else 64 or 32
        int gw = kHThreads;
        {
            const int lo = min(min(s_lo[0], s_lo[1]), min(s_lo[2], s_lo[3]));
            const int hi = max(max(s_hi[0], s_hi[1]), max(s_hi[2], s_hi[3]));
            const int lo01 = min(s_lo[0], s_lo[1]), hi01 = max(s_hi[0], s_hi[1]);
            const int lo23 = min(s_lo[2], s_lo[3]), hi23 = max(s_hi[2], s_hi[3]);
            if (hi - lo > kHB - 16) gw = (max(hi01 - lo01, hi23 - lo23) > kHB - 16) ? 32 : 64;
        }
        const int ngroups = kHThreads / gw;
        const int rstep = kHThreads / gw;
        for (int g = 0; g < ngroups; ++g) {
            const int xg0 = x0 + g * gw;
            if (xg0 >= nx) break;         // uniform: the tile's remaining groups lie past the surface
            if (g > 0) {
                __syncthreads();          // the previous group's convolution has read H
                for (int i = t; i < kHB * L; i += kHThreads) { Hre[i] = (T)0; Him[i] = (T)0; }
                __syncthreads();
            }
            int base;
            {
                const int w0 = g * gw / 32, w1 = w0 + gw / 32;
                int lo = 0x3fffffff, hi = -0x3fffffff;
                for (int k = w0; k < w1; ++k) { lo = min(lo, s_lo[k]); hi = max(hi, s_hi[k]); }
                base = hi >= lo ? lo - (kHB - (hi - lo + 1)) / 2 : 0;
            }
            const int x = xg0 + t % gw;
            int tlo = kHB, thi = -1;
            if (x < nx) {
                const long long g0 = (long long)y0 * nx + x;
                // one facet: into H, or (outside H, non-finite, or an invalid range whose
                // marker bin puts every tap below 0) by the direct path
                auto facet = [&](double s, cplx<T> c) {
                    int bin_d, lut;
                    bin_of(s, bin_d, lut);
                    const int cb = (int)((unsigned)bin_d - (unsigned)base);
                    if ((unsigned)cb < (unsigned)kHB && isfinite(c.re + c.im)) {
                        const int cell = cb * L + lut;
                        atomicAdd(Hre + cell, c.re);
                        atomicAdd(Him + cell, c.im);
                        tlo = min(tlo, cb);
                        thi = max(thi, cb);
                    } else {
                        direct_taps<T>(bin_d, lut, c, sinc, taps, ovs, out, nbins);
                    }
                };
                int r0 = t / gw;
                for (; r0 + (kHRB - 1) * rstep < nrows; r0 += kHRB * rstep) {      // full batches
                    double sr[kHRB];
                    cplx<T> c[kHRB];
#pragma unroll
                    for (int k = 0; k < kHRB; ++k) {
                        const long long gi = g0 + (long long)(r0 + k * rstep) * nx;
                        sr[k] = __ldg(srg + gi);
                        c[k] = load_scene<T, VEC>(scene + gi);
                    }
#pragma unroll
                    for (int k = 0; k < kHRB; ++k) facet(sr[k], c[k]);
                }
                for (; r0 < nrows; r0 += rstep) {                                   // the rest
                    const long long gi = g0 + (long long)r0 * nx;
                    facet(__ldg(srg + gi), load_scene<T, VEC>(scene + gi));
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                tlo = min(tlo, __shfl_xor_sync(0xffffffffu, tlo, o));
                thi = max(thi, __shfl_xor_sync(0xffffffffu, thi, o));
            }
            if (lane == 0) { s_tlo[warp] = tlo; s_thi[warp] = thi; }
            __syncthreads();
            const int clo = min(min(s_tlo[0], s_tlo[1]), min(s_tlo[2], s_tlo[3]));
            const int chi = max(max(s_thi[0], s_thi[1]), max(s_thi[2], s_thi[3]));
            if (chi < clo) continue;      // uniform: nothing landed in H
            // ---- convolution: output bin base + clo - half + m, m < chi - clo + taps; four
            // lanes per output bin, each a quarter of the taps, summed by shuffles ----
            const int nob = chi - clo + taps;
            const int tq = (taps + 3) / 4;
            const int items = nob * 4;
            for (int i0 = 0; i0 < items; i0 += kHThreads) {
                const int i = i0 + t;
                const int m = i >> 2, jq = i & 3;
                T sre = (T)0, sim = (T)0;
                if (i < items) {
                    const int ja = jq * tq, jb = min(taps, ja + tq);
                    for (int j = ja; j < jb; ++j) {
                        const int cell = clo + m - j;          // H bin feeding output m through tap j
                        if (cell < clo || cell > chi) continue;
                        const T *hr = Hre + cell * L, *hi = Him + cell * L;
                        const T *wj = w + j * L;
                        for (int l = 0; l < L; ++l) {
                            sre = fma(wj[l], hr[l], sre);
                            sim = fma(wj[l], hi[l], sim);
                        }
                    }
                }
                sre += __shfl_xor_sync(0xffffffffu, sre, 1);
                sim += __shfl_xor_sync(0xffffffffu, sim, 1);
                sre += __shfl_xor_sync(0xffffffffu, sre, 2);
                sim += __shfl_xor_sync(0xffffffffu, sim, 2);
                const int b = base + clo - half + m;
                if (i < items && jq == 0 && b >= 0 && b < nbins) {
                    if (sre != (T)0) atomicAdd(out + 2 * b, sre);
                    if (sim != (T)0) atomicAdd(out + 2 * b + 1, sim);
                }
            }
        }
    }
}

template <typename T, bool VEC>
static int launch_chan_profile_2d_hist_v(const double *srg, const void *scene, long long ny, long long nx,
                                         double binsize, double min_sr, const float *sinc, int taps, int ovs, T *out,
                                         int nbins, cudaStream_t stream) {
    const size_t smem = hist_smem_bytes<T>(taps, ovs);
    auto kern = chan_profile_2d_hist_kernel<T, VEC>;
    if (ensure_smem((const void *)kern, smem) != cudaSuccess) return OCS_ERR_CUDA;
    const int resident = resident_ctas((const void *)kern, kHThreads, smem);
    if (resident <= 0) return OCS_ERR_CUDA;
    // about one tile per resident CTA: tall tiles amortise the convolution and the global
    // adds of a tile over more facets
    const long long tiles_x = (nx + kHThreads - 1) / kHThreads;
    long long per_col = resident / tiles_x;
    if (per_col < 1) per_col = 1;
    long long rows = (ny + per_col - 1) / per_col;
    if (rows > 1024) rows = 1024;
    if (rows < 1) rows = 1;
    const long long tiles = tiles_x * ((ny + rows - 1) / rows);
    if (tiles > 0x7fffffffLL) return OCS_ERR_SIZE;
    kern<<<(unsigned)tiles, kHThreads, smem, stream>>>(srg, reinterpret_cast<const cplx<T> *>(scene), (int)ny,
                                                        (int)nx, binsize, min_sr, sinc, taps, ovs, out, nbins,
                                                        (int)rows);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

template <typename T>
static int launch_chan_profile_2d_hist(const double *srg, const void *scene, long long ny, long long nx,
                                       double binsize, double min_sr, const float *sinc, int taps, int ovs, T *out,
                                       int nbins, cudaStream_t stream) {
    if (ny > 0x7fffffffLL || nx > 0x7fffffffLL) return OCS_ERR_SIZE;
    if (((uintptr_t)scene & (2 * sizeof(T) - 1)) == 0)
        return launch_chan_profile_2d_hist_v<T, true>(srg, scene, ny, nx, binsize, min_sr, sinc, taps, ovs, out,
                                                      nbins, stream);
    return launch_chan_profile_2d_hist_v<T, false>(srg, scene, ny, nx, binsize, min_sr, sinc, taps, ovs, out, nbins,
                                                   stream);
}

template <typename T>
static int launch_chan_profile_2d_any(const double *srg, const void *scene, long long ny, long long nx,
                                      double binsize, double min_sr, const float *sinc, int taps, int ovs, T *out,
                                      int nbins, cudaStream_t stream) {
    if (taps >= 1 && taps <= 16 && ovs >= 1 && hist_smem_bytes<T>(taps, ovs) <= 40 * 1024)
        return launch_chan_profile_2d_hist<T>(srg, scene, ny, nx, binsize, min_sr, sinc, taps, ovs, out, nbins,
                                              stream);
    if (taps <= 8)
        return launch_chan_profile_2d_regs<T, 12>(srg, scene, ny, nx, binsize, min_sr, sinc, taps, ovs, out, nbins,
                                                  stream);
    return launch_chan_profile_2d_regs<T, 16>(srg, scene, ny, nx, binsize, min_sr, sinc, taps, ovs, out, nbins, stream);
}

// Small host tables carried to the device as kernel parameters: the launch copies them, so the
// caller's memory is free at once and the stream never waits for a pageable copy.
constexpr int kTableFloats = 1000;
struct TableArgs { float v[kTableFloats]; };
__global__ void store_table_kernel(const __grid_constant__ TableArgs a, float *dst, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = a.v[i];
}

}  // namespace ocs

extern "C" int ocs_store_table(float *dst_d, const float *src, int32_t n, void *stream) {
    if (n < 0 || (n > 0 && (!dst_d || !src))) return OCS_ERR_ARG;
    for (int32_t i = 0; i < n; i += ocs::kTableFloats) {
        const int m = n - i < ocs::kTableFloats ? n - i : ocs::kTableFloats;
        ocs::TableArgs a;
        memcpy(a.v, src + i, m * sizeof(float));
        ocs::store_table_kernel<<<(m + 255) / 256, 256, 0, (cudaStream_t)stream>>>(a, dst_d + i, m);
    }
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

extern "C" int ocs_chan_profile_f64(const double *srg, const double *scene, int64_t npts,
                                    double binsize, double min_sr, const float *sinc_vec,
                                    int n_sinc_samples, int sinc_ovs, double *output, int64_t nbins,
                                    void *stream) {
    if (npts < 0 || nbins < 0) return OCS_ERR_ARG;
    if (npts == 0 || nbins == 0) return OCS_OK;
    if (!srg || !scene || !sinc_vec || !output) return OCS_ERR_ARG;
    if (nbins > 0x3fffffff) return OCS_ERR_SIZE;
    const int hb = ocs::flat_grid_bins<double>(n_sinc_samples, sinc_ovs, binsize, (int)nbins);
    if (hb > 0)
        return ocs::launch_chan_profile_flat<double>(srg, scene, npts, binsize, min_sr, sinc_vec, n_sinc_samples, sinc_ovs,
                                                 output, (int)nbins, hb, (cudaStream_t)stream);
    return ocs::launch_chan_profile<double, 16>(srg, scene, 1, npts, binsize, min_sr, sinc_vec,
                                                n_sinc_samples, sinc_ovs, output, (int)nbins,
                                                (cudaStream_t)stream);
}

extern "C" int ocs_chan_profile_rows_f64(const double *srg, const double *scene, int64_t naz,
                                         int64_t npts, double binsize, double min_sr,
                                         const float *sinc_vec, int n_sinc_samples, int sinc_ovs,
                                         double *output, int64_t nbins, void *stream) {
    if (naz < 0 || npts < 0 || nbins < 0) return OCS_ERR_ARG;
    if (naz == 0 || npts == 0 || nbins == 0) return OCS_OK;
    if (!srg || !scene || !sinc_vec || !output) return OCS_ERR_ARG;
    if (nbins > 0x3fffffff) return OCS_ERR_SIZE;
    return ocs::launch_chan_profile<double, 16>(srg, scene, naz, npts, binsize, min_sr, sinc_vec,
                                                n_sinc_samples, sinc_ovs, output, (int)nbins,
                                                (cudaStream_t)stream);
}

extern "C" int ocs_chan_profile_c64(const double *srg, const float *scene, int64_t npts,
                                    double binsize, double min_sr, const float *sinc_vec,
                                    int n_sinc_samples, int sinc_ovs, float *output, int64_t nbins,
                                    void *stream) {
    if (npts < 0 || nbins < 0) return OCS_ERR_ARG;
    if (npts == 0 || nbins == 0) return OCS_OK;
    if (!srg || !scene || !sinc_vec || !output) return OCS_ERR_ARG;
    if (nbins > 0x3fffffff) return OCS_ERR_SIZE;
    const int hb = ocs::flat_grid_bins<float>(n_sinc_samples, sinc_ovs, binsize, (int)nbins);
    if (hb > 0)
        return ocs::launch_chan_profile_flat<float>(srg, scene, npts, binsize, min_sr, sinc_vec, n_sinc_samples, sinc_ovs,
                                                 output, (int)nbins, hb, (cudaStream_t)stream);
    return ocs::launch_chan_profile<float, 16>(srg, scene, 1, npts, binsize, min_sr, sinc_vec,
                                               n_sinc_samples, sinc_ovs, output, (int)nbins,
                                               (cudaStream_t)stream);
}

extern "C" int ocs_chan_profile_2d_f64(const double *srg, const double *scene, int64_t ny, int64_t nx,
                                       double binsize, double min_sr, const float *sinc_vec, int n_sinc_samples,
                                       int sinc_ovs, double *output, int64_t nbins, void *stream) {
    if (ny < 0 || nx < 0 || nbins < 0) return OCS_ERR_ARG;
    if (ny == 0 || nx == 0 || nbins == 0) return OCS_OK;
    if (!srg || !scene || !sinc_vec || !output) return OCS_ERR_ARG;
    if (nbins > 0x3fffffff) return OCS_ERR_SIZE;
    return ocs::launch_chan_profile_2d_any<double>(srg, scene, ny, nx, binsize, min_sr, sinc_vec, n_sinc_samples,
                                                   sinc_ovs, output, (int)nbins, (cudaStream_t)stream);
}

extern "C" int ocs_chan_profile_2d_c64(const double *srg, const float *scene, int64_t ny, int64_t nx,
                                       double binsize, double min_sr, const float *sinc_vec, int n_sinc_samples,
                                       int sinc_ovs, float *output, int64_t nbins, void *stream) {
    if (ny < 0 || nx < 0 || nbins < 0) return OCS_ERR_ARG;
    if (ny == 0 || nx == 0 || nbins == 0) return OCS_OK;
    if (!srg || !scene || !sinc_vec || !output) return OCS_ERR_ARG;
    if (nbins > 0x3fffffff) return OCS_ERR_SIZE;
    return ocs::launch_chan_profile_2d_any<float>(srg, scene, ny, nx, binsize, min_sr, sinc_vec, n_sinc_samples,
                                                  sinc_ovs, output, (int)nbins, (cudaStream_t)stream);
}

