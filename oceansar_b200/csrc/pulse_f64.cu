// Launches of the float64 fine-grid pulse kernel (pulse_f64.cuh): single scenes and the scene
// batch.
#include "pulse_f64.cuh"

namespace ocs {

template <int NOUT, int NPOL, bool XTI>
__global__ void __launch_bounds__(kF64Threads, 2) pulse_f64_kernel(const __grid_constant__ PulseArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const F64Smem<NOUT> sm = f64_smem<NOUT>(smem, kPulseRows);
    grid_wait();
    f64_init<NOUT>(sm, a.sinc);
    double spec_sum = 0.0;
    f64_tile<NOUT, NPOL, XTI>(a, blockIdx.x, a.tile_rows, sm, spec_sum);
    if (a.out0 == 0 && a.do_kodis) block_atomic_sum(spec_sum, &a.nrcs_spec[a.az_step], sm.sred);
}

template <int NOUT, int NPOL, bool XTI>
static int launch_f64(PulseArgs a, cudaStream_t st) {
    const size_t smem = f64_smem_bytes<NOUT>(kPulseRows);
    auto k = pulse_f64_kernel<NOUT, NPOL, XTI>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    const int resident = resident_ctas((const void *)k, kF64Threads, smem);
    if (resident <= 0) return OCS_ERR_CUDA;
    a.tile_rows = tile_rows_for(a.nx, a.ny, kPulseCols, resident, kF64Streams);
    const long long grid = (long long)((a.nx + kPulseCols - 1) / kPulseCols) * ((a.ny + a.tile_rows - 1) / a.tile_rows);
    return launch_pdl(k, dim3((unsigned)grid), kF64Threads, smem, st, a) == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

template <int NOUT>
static int launch_f64_n(const PulseArgs &a, cudaStream_t st) {
    if (a.npol == 2) return a.any_xti ? launch_f64<NOUT, 2, true>(a, st) : launch_f64<NOUT, 2, false>(a, st);
    return a.any_xti ? launch_f64<NOUT, 1, true>(a, st) : launch_f64<NOUT, 1, false>(a, st);
}

int launch_pulse_f64(PulseArgs a, cudaStream_t st) {
    if (a.nout == 1) return launch_f64_n<1>(a, st);
    if (a.nout == 2) return launch_f64_n<2>(a, st);
    return launch_f64_n<4>(a, st);
}

// The batch: one launch covers every live kSlotStd slot's output groups of width NOUT.
template <int NOUT>
__global__ void __launch_bounds__(kF64Threads, 2) batch_pulse_f64_kernel(const __grid_constant__ BatchRef b) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ PulseArgs pa;
    __shared__ int pref[kMaxSlots + 1];
    constexpr int G = 2;
    const int total = scan_slots(b, pref, [](const SlotState &g) {
        int o, w;
        return (slot_live(g) && g.kind == kSlotStd) ? groups_of_class(g.nout, G, NOUT, -1, o, w) * slot_pulse_tiles(g) : 0;
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
    const F64Smem<NOUT> sm = f64_smem<NOUT>(smem, kPulseRowsMax);
    f64_init<NOUT>(sm, pa.sinc);
    double spec_sum = 0.0;
    if (pa.npol == 2) f64_tile<NOUT, 2, true>(pa, tile, g.tile_rows, sm, spec_sum);
    else f64_tile<NOUT, 1, true>(pa, tile, g.tile_rows, sm, spec_sum);
    if (pa.out0 == 0 && pa.do_kodis) block_atomic_sum(spec_sum, &pa.nrcs_spec[pa.az_step], sm.sred);
}

template <int NOUT>
static int batch_f64_n(const BatchRef &b, int grid, cudaStream_t st) {
    const size_t smem = f64_smem_bytes<NOUT>(kPulseRowsMax);
    auto k = batch_pulse_f64_kernel<NOUT>;
    if (ensure_smem((const void *)k, smem) != cudaSuccess) return OCS_ERR_CUDA;
    k<<<grid, kF64Threads, smem, st>>>(b);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

int batch_pulse_f64(const BatchRef &b, int width, int grid, cudaStream_t st) {
    if (width == 1) return batch_f64_n<1>(b, grid, st);
    if (width == 2) return batch_f64_n<2>(b, grid, st);
    return OCS_ERR_ARG;
}

}  // namespace ocs
