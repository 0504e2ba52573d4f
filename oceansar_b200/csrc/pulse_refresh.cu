// The Bragg RCS refresh pass (pulse_refresh.cuh) of a single scene, and the scene batch's
// per-step row tables and refreshes.
#include "pulse_mixed.cuh"
#include "pulse_refresh.cuh"

namespace ocs {

template <typename T>
__global__ void __launch_bounds__(kRefCols) pulse_refresh_kernel(const __grid_constant__ PulseArgs a, int rows) {
    grid_wait();
    refresh_item<T>(a, a.az_now, a.az_step, blockIdx.x, rows);
}

int launch_refresh(const PulseArgs &a, int precision, cudaStream_t st) {
    const int rows = refresh_rows(a.nx, a.ny), grid = refresh_items(a.nx, a.ny, rows);
    auto k = precision == OCS_PREC_F64 ? pulse_refresh_kernel<double> : pulse_refresh_kernel<float>;
    return launch_pdl(k, dim3(grid), kRefCols, 0, st, a, rows) == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

// Items of a slot: its row-table blocks, then (refresh pulses) its refresh items.
template <bool MIXED>
__global__ void __launch_bounds__(kRefCols) batch_pulse_rows_kernel(const __grid_constant__ BatchRef b) {
    using T = typename std::conditional<MIXED, float, double>::type;
    __shared__ int pref[kMaxSlots + 1];
    // the fine-grid slots' tiles evaluate their rows themselves
    const auto row_items = [](const SlotState &g) { return g.kind == kSlotStd ? 0 : (g.ny + kRefCols - 1) / kRefCols; };
    const int total = scan_slots(b, pref, [&](const SlotState &g) {
        if (!slot_live(g)) return 0;
        const bool refresh = (g.flags_tab[g.counter] & kFlagRefresh) && static_cast<const PulseArgs *>(g.pargs)->do_bragg;
        return row_items(g) + (refresh ? refresh_items(g.nx, g.ny, refresh_rows(g.nx, g.ny)) : 0);
    });
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        const int s = find_slot(pref, b.nslots, item);
        const SlotState &g = b.slots[s];
        const PulseArgs &a = *static_cast<const PulseArgs *>(g.pargs);
        const int j = item - pref[s], nr = row_items(g);
        if (j >= nr) {
            refresh_item<T>(a, g.aznow_tab[g.counter], g.counter, j - nr, refresh_rows(g.nx, g.ny));
            continue;
        }
        const int y = j * kRefCols + threadIdx.x;
        if (y < a.ny) {
            // Kirchhoff slots run the float64-range kernel, which reads the float64 table only
            if (MIXED && g.kind != kSlotKa) mix_row(a, g.aznow_tab[g.counter], y);
            else pulse_row(a, g.aznow_tab[g.counter], y);
        }
    }
}

int batch_launch_pulse_rows(const BatchRef &b, int precision, cudaStream_t st) {
    int sms = 0, dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return OCS_ERR_CUDA;
    if (precision == OCS_PREC_MIXED) batch_pulse_rows_kernel<true><<<sms * 4, kRefCols, 0, st>>>(b);
    else batch_pulse_rows_kernel<false><<<sms * 4, kRefCols, 0, st>>>(b);
    return cudaGetLastError() == cudaSuccess ? OCS_OK : OCS_ERR_CUDA;
}

}  // namespace ocs
