// Launches of the float64-range pulse kernel (pulse_core.cuh): the float64 drop-in, and every
// Kirchhoff, DopSCA and SKIM pulse in both precisions; single scenes and the scene batch.
#include "pulse_core.cuh"

namespace ocs {

// One launch covers every live slot's groups of width class NOUT among the slots of its
// pulse-kernel class (MODE = kModeStd: Kodis / Bragg slots, kModeKa: Kirchhoff slots); the
// host sizes the grid for all slots in use and each CTA takes one (slot, group, tile) item.
template <typename T, int NOUT, int S, int MODE = kModeStd>
__global__ void __launch_bounds__(kPulseCols, (sizeof(T) == 4 && NOUT < 4) ? 4 : 2)
batch_pulse_kernel(const __grid_constant__ BatchRef b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ PulseArgs pa;
    __shared__ int pref[kMaxSlots + 1];
    constexpr int G = sizeof(T) == 4 ? 4 : 2;
    constexpr int kind = (MODE & kModeKa) ? kSlotKa : kSlotWide;
    const int total = scan_slots(b, pref, [](const SlotState &g) {
        int o, w;
        return (slot_live(g) && g.kind == kind) ? groups_of_class(g.nout, G, NOUT, -1, o, w) * slot_pulse_tiles(g) : 0;
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
    }
    __syncthreads();
    const PulseSmem<T> sm = pulse_smem<T, NOUT, S, kPulseRowsMax>(smem, kMaxCh);
    build_wtab<T, S>(sm.wtab, pa.sinc, kSincTaps, kSincOvs);
    double spec_sum = 0.0, bragg_sum[2] = {0.0, 0.0};
    pulse_tile<T, NOUT, S, kPulseRowsMax, MODE>(pa, tile, g.tile_rows, sm, spec_sum, bragg_sum);
    pulse_nrcs<T>(pa, sm, spec_sum);
}

template <typename T, int NOUT, int S>
static int launch_pulse(PulseArgs a, cudaStream_t st) {
    const size_t smem = pulse_smem_bytes<T, NOUT, S, kPulseRows>(a.nch);
    auto k = a.sca ? (a.spec_mode != 0 ? pulse_kernel<T, NOUT, S, kModeSca | kModeKa>
                                       : pulse_kernel<T, NOUT, S, kModeSca>)
           : a.skim ? (a.spec_mode != 0 ? pulse_kernel<T, NOUT, S, kModeSkim | kModeKa>
                                        : pulse_kernel<T, NOUT, S, kModeSkim>)
                    : (a.spec_mode != 0 ? pulse_kernel<T, NOUT, S, kModeKa> : pulse_kernel<T, NOUT, S, kModeStd>);
    if (ensure_smem((const void *)k, smem) != cudaSuccess)
        return OCS_ERR_CUDA;
    const int resident = resident_ctas((const void *)k, kPulseCols, smem);
    if (resident <= 0) return OCS_ERR_CUDA;
    a.tile_rows = tile_rows_for(a.nx, a.ny, kPulseCols, resident, 16);
    // SKIM: a tile must not straddle two output rows (ny_integ is a power of two or ny)
    if (a.skim && a.ny_integ < a.ny) {
        a.tile_rows = a.ny_integ;
        while (a.tile_rows > kPulseRows) {
            if (a.tile_rows % 2) return OCS_ERR_ARG;
            a.tile_rows /= 2;
        }
    }
    const long long tiles = (long long)((a.nx + kPulseCols - 1) / kPulseCols) * ((a.ny + a.tile_rows - 1) / a.tile_rows);
    const long long grid = tiles < resident ? tiles : resident;
    k<<<(unsigned)grid, kPulseCols, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

template <typename T, int NOUT, int S, int MODE = kModeStd>
static int batch_pulse_n(const BatchRef &b, int grid, cudaStream_t st) {
    const size_t smem = pulse_smem_bytes<T, NOUT, S, kPulseRowsMax>(kMaxCh);
    auto k = batch_pulse_kernel<T, NOUT, S, MODE>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    k<<<grid, kPulseCols, smem, st>>>(b);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

int launch_pulse_general(const PulseArgs &a, int precision, cudaStream_t st) {
    if (precision == OCS_PREC_F64)
        return a.nout == 1 ? launch_pulse<double, 1, 12>(a, st) : launch_pulse<double, 2, 12>(a, st);
    if (a.nout == 1) return launch_pulse<float, 1, 12>(a, st);
    if (a.nout == 2) return launch_pulse<float, 2, 12>(a, st);
    return launch_pulse<float, 4, 12>(a, st);
}

int batch_pulse_general(const BatchRef &b, int precision, int kind, int width, int grid, cudaStream_t st) {
    if (kind == kSlotKa) {
        // Kirchhoff scenes: float64 ranges and phases in both precisions, as their single-scene
        // pulses run (float32 for the rest in the mixed form)
        if (precision == OCS_PREC_F64) {
            if (width == 1) return batch_pulse_n<double, 1, 12, kModeKa>(b, grid, st);
            if (width == 2) return batch_pulse_n<double, 2, 12, kModeKa>(b, grid, st);
            return OCS_ERR_ARG;
        }
        if (precision == OCS_PREC_MIXED) {
            if (width == 1) return batch_pulse_n<float, 1, 12, kModeKa>(b, grid, st);
            if (width == 2) return batch_pulse_n<float, 2, 12, kModeKa>(b, grid, st);
            if (width == 4) return batch_pulse_n<float, 4, 12, kModeKa>(b, grid, st);
            return OCS_ERR_ARG;
        }
        return OCS_ERR_ARG;
    }
    if (precision == OCS_PREC_F64) {
        if (width == 1) return batch_pulse_n<double, 1, 12>(b, grid, st);
        if (width == 2) return batch_pulse_n<double, 2, 12>(b, grid, st);
    }
    return OCS_ERR_ARG;
}

}  // namespace ocs
