// Launches of the split-range mixed pulse kernels (pulse_mixed.cuh): single scenes and the scene
// batch.
#include "pulse_mixed.cuh"

namespace ocs {

// The mixed form of the batch: every slot's scene passes pulse_split_ok (checked when the
// slot is set) and its tile runs the split-range form of its class (the fine grid, HIST, or
// the register windows of kSlotWide scenes); the raw rows take plain float32 atomics (no
// compensation row).
// Resident CTAs of the fine grid: three (80 registers, some spills) pay for two outputs only
// (58 -> 42 us per step of the six-scene batch; one output 30 -> 36, four 60 -> 71).
template <int NOUT, bool HIST>
__global__ void __launch_bounds__(HIST ? kHistThreads : kMixCols, HIST ? (NOUT == 2 ? 3 : 2) : (NOUT < 4 ? 3 : 2))
batch_pulse_mixed_kernel(const __grid_constant__ BatchRef b) {
    extern __shared__ __align__(128) unsigned char mix_raw[];
    __shared__ PulseArgs pa;
    __shared__ int pref[kMaxSlots + 1];
    constexpr int G = 4;
    const int total = scan_slots(b, pref, [](const SlotState &g) {
        int o, w;
        return (slot_live(g) && g.kind == (HIST ? kSlotStd : kSlotWide))
                   ? groups_of_class(g.nout, G, NOUT, -1, o, w) * slot_pulse_tiles(g) : 0;
    });
    const int item = blockIdx.x;
    if (item >= total) return;
    const int s = find_slot(pref, b.nslots, item);
    const SlotState &g = b.slots[s];
    const int tiles = slot_pulse_tiles(g);
    const int j = item - pref[s];
    const int grp = j / tiles, tile = j - grp * tiles;
    {
        const int *src = static_cast<const int *>(g.pargs);
        int *dst = reinterpret_cast<int *>(&pa);
        for (int i = threadIdx.x; i < (int)(sizeof(PulseArgs) / 4); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int c = g.counter;
        int o = 0, w = 0;
        groups_of_class(g.nout, G, NOUT, grp, o, w);
        pa.out0 = o;
        pa.nout = w;
        pa.az_step = c;
        pa.az_now = g.aznow_tab[c];
        pa.tmod_m = g.tmod_tab[2 * c];
        pa.tmod_p = g.tmod_tab[2 * c + 1];
        pa.raw_row = (long long)c * pa.nbins;
        pa.tile_rows = g.tile_rows;
    }
    double spec_sum = 0.0;
    double *sred;
    // the fast configurations of the single-scene kernel, chosen per CTA from its slot
    const bool fast = pa.do_kodis && pa.do_bragg && pa.npol == 1;
    if constexpr (HIST) {
        const HistSmem<NOUT> sm = hist_smem<NOUT>(mix_raw, kPulseRowsMax);
        hist_init<NOUT>(sm, pa.sinc);
        sred = sm.sred;
        __syncthreads();                  // the pulse's entries of pa
        const bool f = fast && pa.nout == NOUT;
        if (f && !pa.any_xti) mix_hist_tile<NOUT, true, 1>(pa, nullptr, tile, g.tile_rows, sm, spec_sum);
        else if (f) mix_hist_tile<NOUT, true, 2>(pa, nullptr, tile, g.tile_rows, sm, spec_sum);
        else mix_hist_tile<NOUT, true, 0>(pa, nullptr, tile, g.tile_rows, sm, spec_sum);
    } else {
        const MixSmem<NOUT> sm = mix_smem<NOUT>(mix_raw, kMaxCh, kPulseRowsMax);
        build_wtab<float, kMixS>(sm.wtab, pa.sinc, kSincTaps, kSincOvs);
        mix_init<NOUT>(sm);
        sred = sm.sred;
        unsigned rseq = 0;
        bool bad = false;
        const bool f = fast && pa.nout == NOUT;
        if (f && !pa.any_xti)
            mix_tile<NOUT, true, false, 1>(pa, nullptr, nullptr, tile, g.tile_rows, sm, rseq, bad, spec_sum);
        else if (f)
            mix_tile<NOUT, true, false, 2>(pa, nullptr, nullptr, tile, g.tile_rows, sm, rseq, bad, spec_sum);
        else
            mix_tile<NOUT, true, false>(pa, nullptr, nullptr, tile, g.tile_rows, sm, rseq, bad, spec_sum);
    }
    if (pa.out0 == 0 && pa.do_kodis) block_atomic_sum(spec_sum, &pa.nrcs_spec[pa.az_step], sred);
}

template <int NOUT, bool KODIS, int FAST>
static int launch_windows(PulseArgs a, const MixMaps &maps, float *lo_row, cudaStream_t st) {
    const size_t smem = mix_smem_bytes<NOUT>(a.nch, kPulseRows);
    auto k = pulse_mixed_kernel<NOUT, KODIS, FAST>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    const int resident = resident_ctas((const void *)k, kMixCols, smem);
    if (resident <= 0) return OCS_ERR_CUDA;
    a.tile_rows = tile_rows_for(a.nx, a.ny, kMixCols, resident, 16);
    const long long tiles = (long long)((a.nx + kMixCols - 1) / kMixCols) * ((a.ny + a.tile_rows - 1) / a.tile_rows);
    const long long grid = tiles < resident ? tiles : resident;
    k<<<(unsigned)grid, kMixCols, smem, st>>>(a, maps, lo_row);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

template <int NOUT, bool KODIS, int FAST>
static int launch_hist(PulseArgs a, float *lo_row, int most, cudaStream_t st) {
    const size_t smem = hist_smem_bytes<NOUT>(kPulseRows);
    auto k = pulse_mixed_hist_kernel<NOUT, KODIS, FAST>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    const int resident = resident_ctas((const void *)k, kHistThreads, smem);
    if (resident <= 0) return OCS_ERR_CUDA;
    a.tile_rows = tile_rows_for(a.nx, a.ny, kMixCols, resident, kHistStreams);
    if (a.tile_rows > most) a.tile_rows = most;
    // one tile per CTA: with the next pulse's surface passes on a second stream, CTAs start
    // late wherever an SM is still taken, and tiles dealt out in advance would wait for them
    const long long grid = (long long)((a.nx + kMixCols - 1) / kMixCols) * ((a.ny + a.tile_rows - 1) / a.tile_rows);
    return launch_pdl(k, dim3((unsigned)grid), kHistThreads, smem, st, a, lo_row) == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

template <int NOUT, bool KODIS, int FAST>
static int launch_split_f(const PulseArgs &a, const MixMaps &maps, float *lo_row, int hist_rows, cudaStream_t st) {
    return hist_rows > 0 ? launch_hist<NOUT, KODIS, FAST>(a, lo_row, hist_rows, st)
                         : launch_windows<NOUT, KODIS, FAST>(a, maps, lo_row, st);
}

template <int NOUT>
static int launch_split_n(const PulseArgs &a, const MixMaps &maps, float *lo_row, int hist_rows, cudaStream_t st) {
    // the common configurations (one polarisation, every output in this pass, Kodis and Bragg;
    // without (1) or with (2) XTI channels) run instantiations with those fixed
    if (a.do_kodis && a.do_bragg && a.npol == 1 && a.nout == NOUT)
        return a.any_xti ? launch_split_f<NOUT, true, 2>(a, maps, lo_row, hist_rows, st)
                         : launch_split_f<NOUT, true, 1>(a, maps, lo_row, hist_rows, st);
    return a.do_kodis ? launch_split_f<NOUT, true, 0>(a, maps, lo_row, hist_rows, st)
                      : launch_split_f<NOUT, false, 0>(a, maps, lo_row, hist_rows, st);
}

int split_hist_rows(const PulseArgs &a) {
    const double span = tile_span(2.0 * a.kodis.hdx, a.inc_angle, a.binsize);
    return mixed_hist_ok(a.nx, a.ny, a.n_m > a.n_p ? a.n_m : a.n_p, span, a.binsize, hist_least_rows(a.nx, a.ny))
               ? mixed_hist_rows(span) : 0;
}

int launch_pulse_split(const PulseArgs &a, const MixMaps &maps, float *lo_row, int hist_rows, cudaStream_t st) {
    if (a.nout == 1) return launch_split_n<1>(a, maps, lo_row, hist_rows, st);
    if (a.nout == 2) return launch_split_n<2>(a, maps, lo_row, hist_rows, st);
    return launch_split_n<4>(a, maps, lo_row, hist_rows, st);
}

template <int NOUT, bool HIST>
static int batch_split_n(const BatchRef &b, int grid, cudaStream_t st) {
    const size_t smem = HIST ? hist_smem_bytes<NOUT>(kPulseRowsMax) : mix_smem_bytes<NOUT>(kMaxCh, kPulseRowsMax);
    auto k = batch_pulse_mixed_kernel<NOUT, HIST>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    k<<<grid, HIST ? kHistThreads : kMixCols, smem, st>>>(b);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

int batch_pulse_split(const BatchRef &b, int kind, int width, int grid, cudaStream_t st) {
    const bool hist = kind == kSlotStd;
    if (width == 1) return hist ? batch_split_n<1, true>(b, grid, st) : batch_split_n<1, false>(b, grid, st);
    if (width == 2) return hist ? batch_split_n<2, true>(b, grid, st) : batch_split_n<2, false>(b, grid, st);
    if (width == 4) return hist ? batch_split_n<4, true>(b, grid, st) : batch_split_n<4, false>(b, grid, st);
    return OCS_ERR_ARG;
}

}  // namespace ocs
