// Block PCG (pcg_kernel.cuh): the FP64 instantiations.
#include "pcg_kernel.cuh"

namespace gcge {

template void block_pcg_rows<double>(PcgWork &, const SellPattern &, const double *, const double *,
                                     double *, double *, double *, double *, int, int, int, double,
                                     double, bool, bool, cudaStream_t);
}  // namespace gcge
