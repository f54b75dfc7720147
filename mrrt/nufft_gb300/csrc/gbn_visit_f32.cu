// Visit-list spread (gbn_visit.cuh), single precision: a translation unit per precision so
// that they compile in parallel.
#include "gbn_visit.cuh"

namespace gbn {

template cudaError_t launch_visit_count<float>(const VisitBuildParams<float>&, cudaStream_t);
template cudaError_t launch_visit_fill<float>(const VisitBuildParams<float>&, cudaStream_t);
template cudaError_t launch_values<float>(const ValuesParams<float>&, cudaStream_t);
template cudaError_t launch_spread_visits<float>(const VisitParams<float>&, cudaStream_t);

}  // namespace gbn
