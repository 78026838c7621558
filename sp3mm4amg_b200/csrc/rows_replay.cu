// rows_replay.cu -- instantiations and launchers of the replayed row kernels
// (rowreplay.cuh).
#include "rowreplay.cuh"

namespace sp3mm {

namespace {

template <int MODE>
cudaError_t direct_typed(const DirectRowArgs& a, const RowParams& p, const RowGeom& geo,
                         cudaStream_t st) {
    const int tv = a.R.vtype, to = p.c_vt;
    if (MODE == kSymb)
        return launch_row_kernel(k_direct_replay<kSymb, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F64)
        return launch_row_kernel(k_direct_replay<MODE, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F32)
        return launch_row_kernel(k_direct_replay<MODE, double, float>, a, p, geo, st);
    if (tv == SP3MM_F32 && to == SP3MM_F32)
        return launch_row_kernel(k_direct_replay<MODE, float, float>, a, p, geo, st);
    return launch_row_kernel(k_direct_replay<MODE, float, double>, a, p, geo, st);
}

template <int MODE>
cudaError_t pair_typed(const PairRowArgs& a, const RowParams& p, const RowGeom& geo,
                       cudaStream_t st) {
    const int tv = a.A.vtype, to = p.c_vt;
    if (MODE == kSymb)
        return launch_row_kernel(k_pair_replay<kSymb, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F64)
        return launch_row_kernel(k_pair_replay<MODE, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F32)
        return launch_row_kernel(k_pair_replay<MODE, double, float>, a, p, geo, st);
    if (tv == SP3MM_F32 && to == SP3MM_F32)
        return launch_row_kernel(k_pair_replay<MODE, float, float>, a, p, geo, st);
    return launch_row_kernel(k_pair_replay<MODE, float, double>, a, p, geo, st);
}

}  // namespace

size_t replay_bytes(int mode, const ReplayCaps& c, int warps) {
    return replay_place(c, mode != kSymb, warps, 0, nullptr, nullptr, nullptr);
}

cudaError_t launch_direct_replay(const DirectRowArgs& a, const RowParams& p, int mode,
                                 const RowGeom& geo, cudaStream_t st) {
    if (p.nrows <= 0) return cudaSuccess;
    note_launch();
    if (mode == kSymb) return direct_typed<kSymb>(a, p, geo, st);
    if (mode == kNumExact) return direct_typed<kNumExact>(a, p, geo, st);
    return direct_typed<kNumBook>(a, p, geo, st);
}

cudaError_t launch_pair_replay(const PairRowArgs& a, const RowParams& p, int mode,
                               const RowGeom& geo, cudaStream_t st) {
    if (p.nrows <= 0) return cudaSuccess;
    note_launch();
    if (mode == kSymb) return pair_typed<kSymb>(a, p, geo, st);
    if (mode == kNumExact) return pair_typed<kNumExact>(a, p, geo, st);
    return pair_typed<kNumBook>(a, p, geo, st);
}

}  // namespace sp3mm
