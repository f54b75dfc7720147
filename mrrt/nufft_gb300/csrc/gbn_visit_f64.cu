// Visit-list spread (gbn_visit.cuh), double precision: a translation unit per precision so
// that they compile in parallel.
#include "gbn_visit.cuh"

namespace gbn {

template cudaError_t launch_visit_count<double>(const VisitBuildParams<double>&, cudaStream_t);
template cudaError_t launch_visit_fill<double>(const VisitBuildParams<double>&, cudaStream_t);
template cudaError_t launch_values<double>(const ValuesParams<double>&, cudaStream_t);
template cudaError_t launch_spread_visits<double>(const VisitParams<double>&, cudaStream_t);

}  // namespace gbn
