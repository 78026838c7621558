// rows_tiny.cu -- instantiations and launcher of the thread-per-row SpMM
// kernel (rowtiny.cuh).
#include "rowtiny.cuh"

namespace sp3mm {

template <int MODE>
static cudaError_t tiny_typed(const PairRowArgs& a, const RowParams& p, const RowGeom& geo,
                              cudaStream_t st) {
    const int tv = a.A.vtype, to = p.c_vt;
    if (MODE == kSymb)
        return launch_row_kernel(k_pair_tiny<kSymb, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F64)
        return launch_row_kernel(k_pair_tiny<MODE, double, double>, a, p, geo, st);
    if (tv == SP3MM_F64 && to == SP3MM_F32)
        return launch_row_kernel(k_pair_tiny<MODE, double, float>, a, p, geo, st);
    if (tv == SP3MM_F32 && to == SP3MM_F32)
        return launch_row_kernel(k_pair_tiny<MODE, float, float>, a, p, geo, st);
    return launch_row_kernel(k_pair_tiny<MODE, float, double>, a, p, geo, st);
}

cudaError_t launch_pair_tiny(const PairRowArgs& a, const RowParams& p, int mode,
                             cudaStream_t st) {
    if (p.nrows <= 0) return cudaSuccess;
    if (p.S1 < 1 || p.S1 > kTinyProducts) return cudaErrorInvalidValue;
    note_launch();
    RowGeom geo{};
    geo.block = kTinyThreads;
    geo.grid = static_cast<int>((static_cast<long long>(p.nrows) + kTinyThreads - 1) / kTinyThreads);
    geo.smem = tiny_bytes(mode != kSymb, p.S1);
    if (mode == kSymb) return tiny_typed<kSymb>(a, p, geo, st);
    if (mode == kNumExact) return tiny_typed<kNumExact>(a, p, geo, st);
    return tiny_typed<kNumBook>(a, p, geo, st);
}

}  // namespace sp3mm
