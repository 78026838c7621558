// rows_replay.cu -- instantiations and launchers of the replayed row kernels
// (rowreplay.cuh).
#include "rowreplay.cuh"

namespace sp3mm {

namespace {

template <int U, int MODE>
cudaError_t direct_typed(const DirectRowArgs& a, const RowParams& p, const RowGeom& geo,
                         cudaStream_t st) {
    const int tv = a.R.vtype, to = p.c_vt;
    if (MODE == kSymb)
        return launch_row_kernel(k_direct_replay<U, kSymb, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F64)
        return launch_row_kernel(k_direct_replay<U, MODE, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F32)
        return launch_row_kernel(k_direct_replay<U, MODE, double, float>, a, p, geo, st);
    if (tv == SP3MM_F32 && to == SP3MM_F32)
        return launch_row_kernel(k_direct_replay<U, MODE, float, float>, a, p, geo, st);
    return launch_row_kernel(k_direct_replay<U, MODE, float, double>, a, p, geo, st);
}

template <int U, int MODE>
cudaError_t pair_typed(const PairRowArgs& a, const RowParams& p, const RowGeom& geo,
                       cudaStream_t st) {
    const int tv = a.A.vtype, to = p.c_vt;
    if (MODE == kSymb)
        return launch_row_kernel(k_pair_replay<U, kSymb, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F64)
        return launch_row_kernel(k_pair_replay<U, MODE, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F32)
        return launch_row_kernel(k_pair_replay<U, MODE, double, float>, a, p, geo, st);
    if (tv == SP3MM_F32 && to == SP3MM_F32)
        return launch_row_kernel(k_pair_replay<U, MODE, float, float>, a, p, geo, st);
    return launch_row_kernel(k_pair_replay<U, MODE, float, double>, a, p, geo, st);
}

template <int U, int MODE, typename TV, typename TO>
cudaError_t batch_launch(int ctas, size_t smem, cudaStream_t st, const BItem* items,
                         const int4* chunks, const BatchRowParams& p, const BatchReplay& r) {
    if (smem > 48 * 1024) {
        const cudaError_t e = raise_smem_limit(
            reinterpret_cast<const void*>(&k_batch_replay<U, MODE, TV, TO>), smem);
        if (e != cudaSuccess) return e;
    }
    k_batch_replay<U, MODE, TV, TO><<<ctas, 32 * kReplayWarps, smem, st>>>(items, chunks, p, r);
    return cudaGetLastError();
}

template <int U, int MODE>
cudaError_t batch_typed(int tv, int ctas, size_t smem, cudaStream_t st, const BItem* items,
                        const int4* chunks, const BatchRowParams& p, const BatchReplay& r) {
    if (MODE == kSymb)
        return batch_launch<U, kSymb, double, double>(ctas, smem, st, items, chunks, p, r);
    if (tv == SP3MM_F64 && r.to == SP3MM_F64)
        return batch_launch<U, MODE, double, double>(ctas, smem, st, items, chunks, p, r);
    if (tv == SP3MM_F64 && r.to == SP3MM_F32)
        return batch_launch<U, MODE, double, float>(ctas, smem, st, items, chunks, p, r);
    if (tv == SP3MM_F32 && r.to == SP3MM_F32)
        return batch_launch<U, MODE, float, float>(ctas, smem, st, items, chunks, p, r);
    return batch_launch<U, MODE, float, double>(ctas, smem, st, items, chunks, p, r);
}

}  // namespace

namespace {

template <int U>
cudaError_t batch_mode(int mode, int tv, int ctas, size_t smem, cudaStream_t st,
                       const BItem* items, const int4* chunks, const BatchRowParams& p,
                       const BatchReplay& r) {
    if (mode == kSymb) return batch_typed<U, kSymb>(tv, ctas, smem, st, items, chunks, p, r);
    if (mode == kNumExact)
        return batch_typed<U, kNumExact>(tv, ctas, smem, st, items, chunks, p, r);
    return batch_typed<U, kNumBook>(tv, ctas, smem, st, items, chunks, p, r);
}
template <int U>
cudaError_t direct_mode(const DirectRowArgs& a, const RowParams& p, int mode, const RowGeom& geo,
                        cudaStream_t st) {
    if (mode == kSymb) return direct_typed<U, kSymb>(a, p, geo, st);
    if (mode == kNumExact) return direct_typed<U, kNumExact>(a, p, geo, st);
    return direct_typed<U, kNumBook>(a, p, geo, st);
}
template <int U>
cudaError_t pair_mode(const PairRowArgs& a, const RowParams& p, int mode, const RowGeom& geo,
                      cudaStream_t st) {
    if (mode == kSymb) return pair_typed<U, kSymb>(a, p, geo, st);
    if (mode == kNumExact) return pair_typed<U, kNumExact>(a, p, geo, st);
    return pair_typed<U, kNumBook>(a, p, geo, st);
}

}  // namespace

cudaError_t launch_batch_replay(int mode, int tv, int ctas, cudaStream_t st, const BItem* items,
                                const int4* chunks, const BatchRowParams& p,
                                const BatchReplay& r) {
    if (ctas <= 0) return cudaSuccess;
    note_launch();
    const size_t smem = replay_bytes(mode, r.caps, kReplayWarps);
    return replay_unroll(r.caps) == 2
               ? batch_mode<2>(mode, tv, ctas, smem, st, items, chunks, p, r)
               : batch_mode<4>(mode, tv, ctas, smem, st, items, chunks, p, r);
}

size_t replay_bytes(int mode, const ReplayCaps& c, int warps) {
    return replay_place(c, mode != kSymb, warps, 0, nullptr, nullptr, nullptr);
}

cudaError_t launch_direct_replay(const DirectRowArgs& a, const RowParams& p, int mode,
                                 const RowGeom& geo, cudaStream_t st) {
    if (p.nrows <= 0) return cudaSuccess;
    note_launch();
    return replay_unroll(p.rcaps) == 2 ? direct_mode<2>(a, p, mode, geo, st)
                                       : direct_mode<4>(a, p, mode, geo, st);
}

cudaError_t launch_pair_replay(const PairRowArgs& a, const RowParams& p, int mode,
                               const RowGeom& geo, cudaStream_t st) {
    if (p.nrows <= 0) return cudaSuccess;
    note_launch();
    return replay_unroll(p.rcaps) == 2 ? pair_mode<2>(a, p, mode, geo, st)
                                       : pair_mode<4>(a, p, mode, geo, st);
}

}  // namespace sp3mm
