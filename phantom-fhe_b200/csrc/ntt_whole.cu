// ntt_whole.cu - the instantiations and launchers of ntt_whole.cuh (a translation unit of its own: it compiles beside b200fhe.cu)
#include "ntt_whole.cuh"
#include "launch.cuh"

namespace b2 {

template <int LOGN, class Epi, int SRC>
static void fwd(const NttArgs &a, const Epi &epi, uint32_t njobs, uint32_t batch, cudaStream_t s) {
    launch_cl(1u << WholeCfg<LOGN>::LOG_CL, ntt_fwd_whole<LOGN, Epi, SRC>, dim3(njobs << WholeCfg<LOGN>::LOG_CL, batch), WholeCfg<LOGN>::THREADS, whole_smem<LOGN>(), s, a, epi);
}
template <int LOGN>
static void inv(const NttArgs &a, uint32_t njobs, uint32_t batch, cudaStream_t s) {
    launch_cl(1u << WholeCfg<LOGN>::LOG_CL, ntt_inv_whole<LOGN>, dim3(njobs << WholeCfg<LOGN>::LOG_CL, batch), WholeCfg<LOGN>::THREADS, whole_smem<LOGN>(), s, a);
}

void launch_inv_whole(const NttArgs &a, uint32_t njobs, uint32_t batch, cudaStream_t s) {
    switch (a.logN) {
        case 12: inv<12>(a, njobs, batch, s); break;
        case 13: inv<13>(a, njobs, batch, s); break;
        default: inv<14>(a, njobs, batch, s); break;
    }
}
template <class Epi, int SRC>
void launch_fwd_whole(const NttArgs &a, const Epi &epi, uint32_t njobs, uint32_t batch, cudaStream_t s) {
    if constexpr (SRC == 0) {
        if (a.logN == 13) return fwd<13, Epi, SRC>(a, epi, njobs, batch, s);
        if (a.logN == 14) return fwd<14, Epi, SRC>(a, epi, njobs, batch, s);
    }
    fwd<12, Epi, SRC>(a, epi, njobs, batch, s);
}

template void launch_fwd_whole<EpiStore, 0>(const NttArgs &, const EpiStore &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiStore, SRC_WORDS>(const NttArgs &, const EpiStore &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiStore, SRC_CONV>(const NttArgs &, const EpiStore &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiSubFrom, SRC_CONV>(const NttArgs &, const EpiSubFrom &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiSubFromTab, SRC_CONV>(const NttArgs &, const EpiSubFromTab &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiSubMul<false>, SRC_REM | SRC_NEAR>(const NttArgs &, const EpiSubMul<false> &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiSubMul<false>, SRC_REM>(const NttArgs &, const EpiSubMul<false> &, uint32_t, uint32_t, cudaStream_t);
template void launch_fwd_whole<EpiSubMul<false>, SRC_CONV | SRC_REM>(const NttArgs &, const EpiSubMul<false> &, uint32_t, uint32_t, cudaStream_t);

}  // namespace b2
