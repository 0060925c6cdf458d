// Launch of the Hermitian matrix-free Lindblad kernel (lindblad_herm.cu).
#pragma once
#include "stage.cuh"

namespace qg {

template <int DT, int YDT, int EPI>
int launch_lindblad_herm(cudaStream_t st, const qg_lindblad& L, double t, const void* x,
                         const AxpbyArgs& ax, const RkArgs& rk);

}  // namespace qg
