// Plain form: launchers of the single-track kernels (track_f64_impl.cuh).
#include "track_f64_impl.cuh"

namespace ppt {

// (L = 0, the run-time dispatch, has E whatever its maps store.)
template <int ALG, bool COLL, int L>
static void launch_layout(const TrackDev& P, bool rf, int grid, int block, cudaStream_t s) {
    constexpr bool kE = L == 0 || layout_has_e(L);
    const size_t smem = (size_t)P.rf_tab_n * sizeof(double2);
    if (rf && kE) track_f64_kernel<ALG, kE, COLL, L><<<grid, block, smem, s>>>(P);
    else track_f64_kernel<ALG, false, COLL, L><<<grid, block, 0, s>>>(P);
}

template <int ALG, bool COLL>
static void launch_any(const TrackDev& P, bool rf, int grid, int block, cudaStream_t s) {
    switch (f64_single_layout(P)) {
        case kLayFull: launch_layout<ALG, COLL, kLayFull>(P, rf, grid, block, s); break;
        case kLayE: launch_layout<ALG, COLL, kLayE>(P, rf, grid, block, s); break;
        case kLayB: launch_layout<ALG, COLL, kLayB>(P, rf, grid, block, s); break;
        case kLayExEyBz: launch_layout<ALG, COLL, kLayExEyBz>(P, rf, grid, block, s); break;
        case kLayEzBz: launch_layout<ALG, COLL, kLayEzBz>(P, rf, grid, block, s); break;
        case kLayBz: launch_layout<ALG, COLL, kLayBz>(P, rf, grid, block, s); break;
        default: launch_layout<ALG, COLL, 0>(P, rf, grid, block, s);
    }
}

template <int ALG>
static cudaError_t launch_alg(const TrackDev& P, bool rf, bool coll, cudaStream_t s) {
    const int block = pick_block(P.n);
    const int grid = grid_for(P.n, block);
    if (coll) {
        // with a surface only Boris, the default pusher, has kernels for each record layout
        if constexpr (ALG == PPT_ALG_BORIS) launch_any<ALG, true>(P, rf, grid, block, s);
        else launch_layout<ALG, true, 0>(P, rf, grid, block, s);
    } else {
        launch_any<ALG, false>(P, rf, grid, block, s);
    }
    return cudaGetLastError();
}

int launch_track_f64(const TrackDev& P, int algorithm, bool rf, bool coll, cudaStream_t s) {
    cudaError_t e;
    switch (algorithm) {
        case PPT_ALG_LEAPFROG: e = launch_alg<PPT_ALG_LEAPFROG>(P, rf, coll, s); break;
        case PPT_ALG_BORIS: e = launch_alg<PPT_ALG_BORIS>(P, rf, coll, s); break;
        case PPT_ALG_RK4: e = launch_alg<PPT_ALG_RK4>(P, rf, coll, s); break;
        case PPT_ALG_YOSHIDA: e = launch_alg<PPT_ALG_YOSHIDA>(P, rf, coll, s); break;
        case PPT_ALG_VAY_REL: e = launch_alg<PPT_ALG_VAY_REL>(P, rf, coll, s); break;
        case PPT_ALG_RK4_REL: e = launch_alg<PPT_ALG_RK4_REL>(P, rf, coll, s); break;
        case PPT_ALG_YOSHIDA_REL: e = launch_alg<PPT_ALG_YOSHIDA_REL>(P, rf, coll, s); break;
        case PPT_ALG_BORIS_REL: e = launch_alg<PPT_ALG_BORIS_REL>(P, rf, coll, s); break;
        case PPT_ALG_VAY: e = launch_alg<PPT_ALG_VAY>(P, rf, coll, s); break;
        default: return fail(PPT_ERR_ARG, "unknown algorithm");
    }
    if (e != cudaSuccess) return cuda_fail(e, "track_f64_kernel launch");
    return PPT_OK;
}

}  // namespace ppt
