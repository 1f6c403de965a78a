// Explicit instantiation of the stream kernel for VALUE_TYPE double; a translation
// unit of its own, so that the build compiles it beside the other kernels.
#include "kernels_stream.cuh"

namespace capsp {

template cudaError_t launch_stream_solve<double>(const StreamArgs<double> &, bool, bool, int, int, cudaStream_t);
template cudaError_t launch_stream_layout<double>(const StreamBuild<double> &, cudaStream_t);
template cudaError_t launch_stream_values<double>(const StreamBuild<double> &, const int *, const double *, double *, double *, int *,
                                               cudaStream_t);

}  // namespace capsp
