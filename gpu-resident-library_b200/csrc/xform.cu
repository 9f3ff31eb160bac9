#include "xform.cuh"

#include "devonce.hpp"

namespace {

// One transform with column tiles of W columns (ntt::narrow_tiles).
template <int LOGN, bool SINGLE, int W>
cudaError_t launch_w(const xf::Job* jobs, const xf::Job& o, int njobs, bool inverse, cudaStream_t s) {
    using G = ntt::Geo<LOGN, W>;
    static gfx::DeviceOnce attrs;   // shared-memory limits, once per device
    attrs([] {
        cudaFuncSetAttribute(xf::k_fwd_col<LOGN, SINGLE, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::COL_SMEM);
        cudaFuncSetAttribute(xf::k_inv_col<LOGN, SINGLE, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::COL_SMEM);
        cudaFuncSetAttribute(xf::k_fwd_row<LOGN, SINGLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
        cudaFuncSetAttribute(xf::k_inv_row<LOGN, SINGLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
    });
    auto run = [&](auto* kernel, bool after, unsigned grid, unsigned block, size_t smem) {
        return gfx::chain_launch(kernel, after, grid, block, smem, s, jobs, o) == cudaSuccess;
    };
    const unsigned col = njobs * G::COL_TILES, row = njobs * G::ROW_TILES;
    if (!inverse) {
        if (run(xf::k_fwd_col<LOGN, SINGLE, W>, false, col, G::COL_THREADS, G::COL_SMEM))
            run(xf::k_fwd_row<LOGN, SINGLE>, true, row, G::ROW_THREADS, G::ROW_SMEM);
    } else {
        if (run(xf::k_inv_row<LOGN, SINGLE>, false, row, G::ROW_THREADS, G::ROW_SMEM))
            run(xf::k_inv_col<LOGN, SINGLE, W>, true, col, G::COL_THREADS, G::COL_SMEM);
    }
    return cudaGetLastError();   // of either launch
}

template <int LOGN, bool SINGLE>
cudaError_t launch_t(const xf::Job* jobs, const xf::Job* one, int njobs, bool inverse, cudaStream_t s) {
    const xf::Job o = one ? *one : xf::Job{};
    return ntt::narrow_tiles<LOGN>(njobs, gfx::current_sm_count())
               ? launch_w<LOGN, SINGLE, ntt::COL_NARROW>(jobs, o, njobs, inverse, s)
               : launch_w<LOGN, SINGLE, ntt::COL_WIDE>(jobs, o, njobs, inverse, s);
}

template <int LOGN, int W>
cudaError_t launch_lift_w(const xf::Job* jobs, int njobs, cudaStream_t s) {
    using G = ntt::Geo<LOGN, W>;
    static gfx::DeviceOnce attrs;
    attrs([] {
        cudaFuncSetAttribute(xf::k_fwd_col_lift<LOGN, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::COL_SMEM);
        cudaFuncSetAttribute(xf::k_fwd_row<LOGN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::ROW_SMEM);
    });
    if (gfx::chain_launch(xf::k_fwd_col_lift<LOGN, W>, false, njobs * G::COL_TILES, G::COL_THREADS, G::COL_SMEM, s,
                          jobs) == cudaSuccess)
        gfx::chain_launch(xf::k_fwd_row<LOGN, false>, true, njobs * G::ROW_TILES, G::ROW_THREADS, G::ROW_SMEM, s, jobs,
                          xf::Job{});
    return cudaGetLastError();   // of either launch
}

template <int LOGN>
cudaError_t launch_lift(const xf::Job* jobs, int njobs, cudaStream_t s) {
    return ntt::narrow_tiles<LOGN>(njobs, gfx::current_sm_count()) ? launch_lift_w<LOGN, ntt::COL_NARROW>(jobs, njobs, s)
                                                                   : launch_lift_w<LOGN, ntt::COL_WIDE>(jobs, njobs, s);
}

}  // namespace

bool xf_supported_logn(int logn) { return logn >= 9 && logn <= 16; }

cudaError_t xf_launch_ntt_lift(const xf::Job* jobs, int njobs, int logn, cudaStream_t s) {
    if (njobs <= 0) return cudaSuccess;
    switch (logn) {
        case 9: return launch_lift<9>(jobs, njobs, s);
        case 10: return launch_lift<10>(jobs, njobs, s);
        case 11: return launch_lift<11>(jobs, njobs, s);
        case 12: return launch_lift<12>(jobs, njobs, s);
        case 13: return launch_lift<13>(jobs, njobs, s);
        case 14: return launch_lift<14>(jobs, njobs, s);
        case 15: return launch_lift<15>(jobs, njobs, s);
        case 16: return launch_lift<16>(jobs, njobs, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t xf_launch_ntt(const xf::Job* jobs, const xf::Job* one, int njobs, int logn, bool inverse,
                          cudaStream_t s) {
    if (njobs <= 0) return cudaSuccess;
    switch (logn) {
        case 9: return one ? launch_t<9, true>(jobs, one, njobs, inverse, s) : launch_t<9, false>(jobs, one, njobs, inverse, s);
        case 10: return one ? launch_t<10, true>(jobs, one, njobs, inverse, s) : launch_t<10, false>(jobs, one, njobs, inverse, s);
        case 11: return one ? launch_t<11, true>(jobs, one, njobs, inverse, s) : launch_t<11, false>(jobs, one, njobs, inverse, s);
        case 12: return one ? launch_t<12, true>(jobs, one, njobs, inverse, s) : launch_t<12, false>(jobs, one, njobs, inverse, s);
        case 13: return one ? launch_t<13, true>(jobs, one, njobs, inverse, s) : launch_t<13, false>(jobs, one, njobs, inverse, s);
        case 14: return one ? launch_t<14, true>(jobs, one, njobs, inverse, s) : launch_t<14, false>(jobs, one, njobs, inverse, s);
        case 15: return one ? launch_t<15, true>(jobs, one, njobs, inverse, s) : launch_t<15, false>(jobs, one, njobs, inverse, s);
        case 16: return one ? launch_t<16, true>(jobs, one, njobs, inverse, s) : launch_t<16, false>(jobs, one, njobs, inverse, s);
        default: return cudaErrorInvalidValue;
    }
}
