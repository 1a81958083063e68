// Forward entry point of the wavefront scan: one fused kernel, y written directly.
#include "launch.cuh"
#include "sweep_pairs.cuh"
#include "wave_fwd.cuh"

namespace m2d {

// Few images: several CTAs per image.
template <typename io_t, int C, bool VEC, bool ACT, int COLS>
__global__ void __launch_bounds__(256, 1) m2d_fwd_wave_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    wave_forward<io_t, C, VEC, ACT ? kReadoutGelu : kReadout, COLS>(a, reinterpret_cast<char*>(smem));
}

// Batch mode (one CTA per image and channel group): the sweep written as nested loops.
template <typename io_t, bool VEC, bool ACT>
__global__ void __launch_bounds__(kPairWarps * 32, 2) m2d_fwd_kernel(const ScanArgs a) {
    extern __shared__ float4 smem[];
    const PairLane ln(a);
    const unsigned params = begin_pairs<io_t>(a, smem, pairs_fwd_smem_bytes(ln.nwarps), ln);
    const int y_ch = ln.ch0 + (ln.nq & 1);
    forward_pairs<io_t, float, VEC, false, ACT, false>(a, smem_u32(smem), params, y_ch < a.E ? load_D<io_t>(a, y_ch) : 0.f);
}

// The status word and, where CTAs of a wave launch read each other's, the boundary rows behind it.
static size_t cleared_bytes(const m2d_scan_desc* d, const Plan& pl) {
    return kStatusBytes + (pl.wave && pl.chain > 1 ? wave_edge_bytes(d, pl, false) : 0);
}

template <typename io_t>
static int launch_fwd(const m2d_scan_desc* d, const Plan& pl, bool vec, char* ws, cudaStream_t st) {
    ScanArgs a;
    fill_common_args(a, d, pl);
    a.y = d->y;
    a.status = reinterpret_cast<int*>(ws);
    a.ring = reinterpret_cast<float4*>(ws + kStatusBytes);
    const size_t zero = pl.wave && pl.chain > 1 ? cleared_bytes(d, pl) : sizeof(int);
    if (!(d->flags & M2D_SCAN_WS_CLEARED) && cudaMemsetAsync(ws, 0, zero, st) != cudaSuccess) return M2D_ERR_LAUNCH;
    if (!pl.wave) {
        auto pick = [&](auto act) {
            constexpr bool ACT = decltype(act)::value;
            return vec ? m2d_fwd_kernel<io_t, true, ACT> : m2d_fwd_kernel<io_t, false, ACT>;
        };
        return launch_sweep_kernel(a.act ? pick(std::true_type{}) : pick(std::false_type{}), a, pl, st);
    }
    a.bnd = reinterpret_cast<float4*>(ws + kStatusBytes);
    a.bnd_rows = wave_rows(pl, false);
    Plan p = pl;
    p.smem = pl.wave == 4 ? WaveSmem<io_t, 4, false>::kBytes : WaveSmem<io_t, 2, false>::kBytes;
    auto pick = [&](auto act) {
        constexpr bool ACT = decltype(act)::value;
        if (edge_pairs(d, pl, sizeof(io_t)))
            return vec ? m2d_fwd_wave_kernel<io_t, 4, true, ACT, 2> : m2d_fwd_wave_kernel<io_t, 4, false, ACT, 2>;
        return pl.wave == 4 ? (vec ? m2d_fwd_wave_kernel<io_t, 4, true, ACT, kChunk> : m2d_fwd_wave_kernel<io_t, 4, false, ACT, kChunk>)
                            : (vec ? m2d_fwd_wave_kernel<io_t, 2, true, ACT, kChunk> : m2d_fwd_wave_kernel<io_t, 2, false, ACT, kChunk>);
    };
    return launch_sweep_kernel(a.act ? pick(std::true_type{}) : pick(std::false_type{}), a, p, st);
}

int launch_forward(const m2d_scan_desc* d, const Plan& pl, char* scratch, cudaStream_t st) {
    const bool vec = vector_ok(d, false);
    return d->dtype == M2D_F32 ? launch_fwd<float>(d, pl, vec, scratch, st) : launch_fwd<__nv_bfloat16>(d, pl, vec, scratch, st);
}

}  // namespace m2d

extern "C" uint64_t m2d_scan_fwd_workspace(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, false, false) != M2D_OK) return 0;
    return m2d::plan_fwd(d).scratch;
}

extern "C" uint64_t m2d_scan_fwd_cleared(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, false, false) != M2D_OK) return 0;
    return m2d::cleared_bytes(d, m2d::plan_fwd(d));
}

extern "C" int64_t m2d_scan_fwd_status_offset(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, false, false) != M2D_OK) return -1;
    return 0;
}

extern "C" int m2d_scan_fwd_chain(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, false, false) != M2D_OK) return 0;
    return m2d::plan_fwd(d).chain;
}

extern "C" int m2d_scan_fwd_edge_columns(const m2d_scan_desc* d) {
    if (m2d::check_desc(d, false, false) != M2D_OK) return 0;
    const m2d::Plan p = m2d::plan_fwd(d);
    return p.chain < 2 ? 0 : m2d::edge_pairs(d, p, d->dtype == M2D_F32 ? sizeof(float) : sizeof(__nv_bfloat16)) ? 2 : m2d::kChunk;
}

extern "C" int m2d_scan_chain_bound(int want, int nbands, int steps_per_row, int rows_per_band) {
    if (nbands < 1 || steps_per_row < 1 || rows_per_band < 1) return 0;
    return m2d::bound_chain(want, nbands, steps_per_row, rows_per_band);
}

extern "C" int m2d_scan_fwd(const m2d_scan_desc* d, void* stream) {
    int rc = m2d::check_desc(d, false, true);
    if (rc != M2D_OK) return rc;
    if (!d->y) return M2D_ERR_NULL;
    const m2d::Plan pl = m2d::plan_fwd(d);
    if (!d->workspace || d->workspace_bytes < pl.scratch || (reinterpret_cast<uintptr_t>(d->workspace) & 255))
        return M2D_ERR_WORKSPACE;
    return m2d::launch_forward(d, pl, static_cast<char*>(d->workspace), static_cast<cudaStream_t>(stream));
}
